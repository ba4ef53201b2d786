// The IISPH gather phases on stored kernel gradients (here the 3D ones with one
// thread per owner; fs_gather.cuh has those with eight, 2D and 3D).
//
// The bit-exact and FP64 modes evaluate gradW by an IEEE square root and four
// divisions, more than 60 of a pair's 90 instructions, and the positions they
// come from do not change until the integration. The first loop, which needs
// every gradient for the viscosity, stores it with the neighbor's mass beside
// the list entry, slot-major like the list, so a warp writes and reads whole
// lines; the second loop and the pressure iterations read it back and gather
// only the field they are after. The values and the order of the sums are
// those of the functions in fs_solvers.cuh, so the results are the same bit
// for bit. 33 neighbors of 100,000 owners are 53 MB in FP32, which L2 holds.
//
// (In the fast mode's tile passes the same costs more traffic than it saves
// instructions; there the gradient is one rsqrt and no division.)
//
// Measured on a B200, a pressure iteration evaluated and from stored gradients:
// bit-exact mode 78 -> 40 us at 100,000 fluid particles, 512 -> 307 at a million;
// FP64 275 -> 147 at 250,047, 1,034 -> 464 at a million. The first loop's stores
// cost it 8 % and 5 %.
#pragma once

#include "fs_common.cuh"
#include "fs_solvers.cuh"

namespace fsb {

// gradients of list entry q of owner k at [q * stride + k] (Lists::stride): x, y, z, the neighbor's mass
template <typename R> struct Gradients {
    V4<R>* FSB_R g;
};

// Visits owner k's list in order, handing use(entry, gradient and mass,
// load(sorted index)); the loads of a batch are in flight together.
template <typename R, typename Load, typename Use>
__device__ __forceinline__ void for_gradients(const Lists& L, const Gradients<R>& G, int64_t k, Load&& load, Use&& use) {
    const uint32_t n = L.size(k);
    for (uint32_t q = 0; q < n; q += kBatch) {
        uint32_t e[kBatch];
        V4<R> g[kBatch];
        decltype(load(0u)) v[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; b++) {
            const int64_t at = (int64_t)min(q + b, n - 1) * L.stride + k;
            e[b] = FSB_LDG(&L.nbr[at]);
            g[b] = G.g[at];
        }
#pragma unroll
        for (int b = 0; b < kBatch; b++) v[b] = load(e[b] & kIndexMask);
#pragma unroll
        for (int b = 0; b < kBatch; b++)
            if (q + b < n) use(e[b], g[b], v[b]);
    }
}

template <typename R, bool KAHAN, bool SPLIT>
__global__ void __launch_bounds__(128) k_cached_iisph3d_l1(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                           Gradients<R> G, const StepScalars* FSB_R sc,
                                                           const int* FSB_R status) {
    phase_begins(s.phase_at, 1);
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n || *status) return;
    iisph3d_l1_one<R, KAHAN, SPLIT>(k, s, L, c, (R)sc->dt, [&](uint32_t q, const V3<R>& g, const V4<R>& pj) {
        G.g[(int64_t)q * L.stride + k] = v4<R>(g, pj.w);
    });
}

// iisph3d_l2_one
template <typename R, bool KAHAN, bool TWO_PASS>
__global__ void __launch_bounds__(128) k_cached_iisph3d_l2(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                           Gradients<R> G, const StepScalars* FSB_R sc,
                                                           const int* FSB_R status) {
    phase_begins(s.phase_at, 2);
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n || *status || s.type[k] != FS_TYPE_NORMAL) return;
    const R dt = (R)sc->dt;
    const R mk = s.pos[k].w;
    const V3<R> vsk = xyz<R>(s.vstar[k]);
    Acc<R, KAHAN> contrib, mg2;
    Acc3<R, KAHAN> inner, mg;
    for_gradients<R>(L, G, k, [&](uint32_t j) { return s.vstar[j]; }, [&](uint32_t e, const V4<R>& g4, const V4<R>& vsj) {
        const V3<R> g = xyz<R>(g4);
        const R m = g4.w;
        if (!(e & kBoundaryBit)) {
            contrib.add(m * dotf<KAHAN>(vsk - xyz<R>(vsj), g));
            inner.sub((KAHAN ? m * c.inv_rho0_sq : m / c.rho0_sq) * g);
            if (!TWO_PASS) mg2.add(m * dotf<KAHAN>(g, g));
        } else {
            contrib.add(m * dotf<KAHAN>(vsk, g));
            const R w = c.single_layer ? c.two_gamma * m : R(2) * m;
            inner.sub((KAHAN ? w * c.inv_rho0_sq : w / c.rho0_sq) * g);
        }
        if (!TWO_PASS) mg.add(m * g);
    });
    const R source = (c.rest_density - s.rho[k]) - dt * contrib.get();
    const V3<R> in = inner.get();
    R diag;
    if (TWO_PASS) {
        Acc<R, KAHAN> d;
        const R mi = mk / c.rho0_sq;
        for_gradients<R>(L, G, k, [](uint32_t) { return 0; }, [&](uint32_t e, const V4<R>& g4, int) {
            const V3<R> g = xyz<R>(g4);
            d.add(g4.w * dot(in, g));
            if (!(e & kBoundaryBit)) d.add(g4.w * dot(mi * (-g), g));
        });
        diag = d.get() * (dt * dt);
    } else {
        diag = (dot(in, mg.get()) - (mk / c.rho0_sq) * mg2.get()) * (dt * dt);
    }
    s.vstar[k] = v4<R>(vsk, source);
    s.anp[k].w = diag;
}

// iisph3d_pressure_acc_one
template <typename R, bool KAHAN>
__global__ void __launch_bounds__(128) k_cached_iisph3d_pressure_acc(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                                     Gradients<R> G, const StepScalars* FSB_R sc,
                                                                     const int* FSB_R status) {
    phase_begins(s.phase_at, 3);
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n || *status || sc->done || s.type[k] != FS_TYPE_NORMAL) return;
    const R pk = s.p[k], qk = pk / c.rho0_sq;
    Acc3<R, KAHAN> pa;
    for_gradients<R>(L, G, k, [&](uint32_t j) { return s.p[j]; }, [&](uint32_t e, const V4<R>& g4, R pj) {
        const V3<R> g = xyz<R>(g4);
        const R m = g4.w;
        if (KAHAN) {
            const R f = !(e & kBoundaryBit) ? m * (pk + pj) : (c.single_layer ? c.two_gamma : R(2)) * m * pk;
            pa.sub((f * c.inv_rho0_sq) * g);
        } else if (!(e & kBoundaryBit)) {
            pa.sub((m * (qk + pj / c.rho0_sq)) * g);
        } else if (c.single_layer) {
            pa.sub(((((c.gamma * m) * R(2)) * pk) / c.rho0_sq) * g);
        } else {
            pa.sub((((m * R(2)) * pk) / c.rho0_sq) * g);
        }
    });
    s.acc[k] = v4<R>(pa.get(), R(0));
}

// iisph3d_pressure_update_one
template <typename R, bool KAHAN>
__global__ void __launch_bounds__(128) k_cached_iisph3d_pressure_update(int64_t n, State<R> s, Lists L,
                                                                        SolverConsts<R> c, Gradients<R> G,
                                                                        StepScalars* FSB_R sc,
                                                                        const int* FSB_R status) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (*status || sc->done) return;
    ErrPart o;
    if (k < n && s.type[k] == FS_TYPE_NORMAL) {
        const V3<R> ak = xyz<R>(s.acc[k]);
        Acc<R, KAHAN> ap;
        for_gradients<R>(L, G, k, [&](uint32_t j) { return s.acc[j]; },
                         [&](uint32_t e, const V4<R>& g4, const V4<R>& aj) {
            const V3<R> g = xyz<R>(g4);
            if (!(e & kBoundaryBit)) ap.add(g4.w * dotf<KAHAN>(ak - xyz<R>(aj), g));
            else ap.add(g4.w * dotf<KAHAN>(ak, g));
        });
        o = iisph3d_pressure_update_tail<R>(k, s, c, (R)sc->dt, ak, ap.get(), s.vstar[k], s.anp[k].w, s.p[k]);
    }
    reduce_err_parts(o, sc);
}

}  // namespace fsb
