// The gather phases of fs_solvers.cuh with kGroup threads per owner.
//
// With one thread per owner a phase is a serial chain: 20 to 33 neighbors, each
// with gathers, a square root and divisions, on as few threads as there are
// particles. 2,500 owners are 20 blocks of four warps, and a 2D SESPH force
// pass took 20 us of which almost all was that chain's latency; at 100,000
// owners the device was still a quarter busy. Here the threads of a group take
// the list's entries kGroup at a time, a window of kWindow entries in flight
// together, and write every entry's terms to shared memory; then one thread per
// sum adds its terms in list order. So each sum is the one the single thread
// forms, bit for bit, plain or compensated, and only its terms are computed
// side by side. The formulas and their order are those of the functions in
// fs_solvers.cuh (the reference lines stand there).
//
// With many owners the lanes that idle while one of them adds cost more than the
// latency: fs_api.cu (grouped) has the sizes and both sides' times.
#pragma once

#include "fs_cached.cuh"
#include "fs_common.cuh"
#include "fs_solvers.cuh"

namespace fsb {

constexpr int kGroup = 8;            // threads per owner
constexpr int kWindow = 32;          // entries whose terms are in shared memory at a time
constexpr int kGroupThreads = 128;   // 16 owners per block
constexpr int kGroupsPerBlock = kGroupThreads / kGroup;

inline unsigned group_grid(int64_t owners) {
    const int64_t g = (owners + kGroupsPerBlock - 1) / kGroupsPerBlock;
    return (unsigned)(g > 1 ? g : 1);
}

// one group's terms, a row per sum (rows start in different banks)
template <typename R, int NC> struct alignas(16) GroupRows {
    R v[NC][kWindow + 4];
};

template <int G = kGroup> __device__ __forceinline__ int group_lane() { return (int)(threadIdx.x & (G - 1)); }
__device__ __forceinline__ int64_t group_owner() {
    return blockIdx.x * (int64_t)kGroupsPerBlock + threadIdx.x / kGroup;
}

// Adds the terms of the first n entries of owner k's list to the sums: lane c
// of the group holds sum c in acc. load(j, at): the fields of neighbor j, the
// entry lying at `at` in the lists (-1: none, j is then 0); term(entry, fields,
// t): the entry's NC terms, and which of them count: bit 0 for t[0 .. H), bit 1
// for t[H .. NC). INTERLEAVED: two terms per entry of one
// sum, t[0] then t[1], held by lane 0. Every thread of the warp calls it.
template <int NC, int H, bool INTERLEAVED = false, typename R, bool KAHAN, typename Load, typename Term>
__device__ __forceinline__ void group_sum(const Lists& L, int64_t k, uint32_t n, GroupRows<R, NC>& rows,
                                          Acc<R, KAHAN>& acc, Load&& load, Term&& term) {
    constexpr int kRounds = kWindow / kGroup;
    const int g = group_lane();
    const unsigned all = 0xffffffffu, shift = threadIdx.x & 31u & ~(unsigned)(kGroup - 1);
    const uint32_t most = __reduce_max_sync(all, n);
    for (uint32_t base = 0; base < most; base += kWindow) {
        uint32_t e[kRounds];
        decltype(load(0u, (int64_t)0)) d[kRounds];
        int64_t at[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
            const uint32_t q = base + r * kGroup + g;
            at[r] = q < n ? (int64_t)q * L.stride + k : -1;
            e[r] = q < n ? FSB_LDG(&L.nbr[at[r]]) : 0u;
        }
#pragma unroll
        for (int r = 0; r < kRounds; r++) d[r] = load(e[r] & kIndexMask, at[r]);
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
            R t[NC];
            const unsigned ok = term(e[r], d[r], t);
            const bool in = base + r * kGroup + g < n;
#pragma unroll
            for (int c = 0; c < NC; c++) rows.v[c][r * kGroup + g] = t[c];
            constexpr unsigned kMask = (1u << kGroup) - 1u;
            lo |= ((__ballot_sync(all, in && (ok & 1u)) >> shift) & kMask) << (r * kGroup);
            if (H < NC) hi |= ((__ballot_sync(all, in && (ok & 2u)) >> shift) & kMask) << (r * kGroup);
        }
        __syncwarp();
        if (g < (INTERLEAVED ? 1 : NC)) {
            const R* row = rows.v[g];
            const uint32_t mask = INTERLEAVED ? lo | hi : (H < NC && g >= H ? hi : lo);
            const int m = 32 - __clz((int)mask);
#pragma unroll 4
            for (int i = 0; i < m; i++) {
                if (INTERLEAVED) {
                    if ((lo >> i) & 1u) acc.add(row[i]);
                    if ((hi >> i) & 1u) acc.add(rows.v[NC - 1][i]);
                } else {
                    if ((mask >> i) & 1u) acc.add(row[i]);
                }
            }
        }
        __syncwarp();
    }
}
// sum c of the group, in every thread
template <typename R, bool KAHAN> __device__ __forceinline__ R group_total(const Acc<R, KAHAN>& acc, int c) {
    return __shfl_sync(0xffffffffu, acc.get(), c, kGroup);
}
template <typename R, bool KAHAN> __device__ __forceinline__ V3<R> group_total3(const Acc<R, KAHAN>& acc, int c) {
    return v3<R>(group_total(acc, c), group_total(acc, c + 1), group_total(acc, c + 2));
}

// neighbor fields
template <typename R> struct GPos {
    V4<R> x;
};
template <typename R> struct GPosVec {
    V4<R> x, v;
};
template <typename R> struct GPosScalar {
    V4<R> x;
    R a;
};
template <typename R> struct GVisc {
    V4<R> x, v;
    R rho;
    int64_t at;
};
template <typename R> struct GForce {
    V4<R> x, v;
    R rho, p;
};

// CACHED: the stored gradient and mass of the entry (fs_cached.cuh) instead of
// the neighbor's position and mass; then gradW of either
template <bool CACHED, typename R>
__device__ __forceinline__ V4<R> position_or_gradient(const State<R>& s, const Gradients<R>& G, uint32_t j, int64_t at) {
    return CACHED ? G.g[at < 0 ? 0 : at] : s.pos[j];
}
template <bool CACHED, bool KAHAN, typename R>
__device__ __forceinline__ V3<R> gradient_of(const SolverConsts<R>& c, V3<R> xk, const V4<R>& x) {
    return CACHED ? xyz<R>(x) : c.kern.template grad<KAHAN>(xk - xyz<R>(x));
}

// the viscosity term of neighbor (xj, vj, rj) without the factor 2 nu
// (viscosity() in fs_solvers.cuh); false where the density is 0
template <typename R, bool KAHAN>
__device__ __forceinline__ bool viscosity_term(const SolverConsts<R>& c, V3<R> xij, V3<R> g, V3<R> vij, R m, R rj,
                                               R* t) {
    if (rj == R(0)) {
        t[0] = t[1] = t[2] = R(0);
        return false;
    }
    const R f = KAHAN ? fdiv<true>(m * dotf<true>(vij, xij), rj * (dotf<true>(xij, xij) + c.visc_eps))
                      : (m / rj) * (dot(vij, xij) / (dot(xij, xij) + c.visc_eps));
    const V3<R> v = f * g;
    t[0] = v.x;
    t[1] = v.y;
    t[2] = v.z;
    return true;
}
template <typename R> __device__ __forceinline__ void put3(R* t, V3<R> v) {
    t[0] = v.x;
    t[1] = v.y;
    t[2] = v.z;
}

// ---------------------------------------------------------------------------
// density sums: SESPH (with the pressure), IISPH 3D and 2D (split first loop)
// ---------------------------------------------------------------------------
// GAMMA: boundary neighbors weighted by gamma_1 in the single-layer model (3D)
template <typename R, bool KAHAN, bool GAMMA>
__device__ __forceinline__ R group_density(int64_t k, uint32_t n, V3<R> xk, const State<R>& s, const Lists& L,
                                           const SolverConsts<R>& c, GroupRows<R, 1>& rows) {
    Acc<R, KAHAN> acc;
    group_sum<1, 1>(L, k, n, rows, acc, [&](uint32_t j, int64_t) { return GPos<R>{s.pos[j]}; },
                    [&](uint32_t e, const GPos<R>& d, R* t) {
                        R m = d.x.w;
                        if (GAMMA && c.single_layer && (e & kBoundaryBit)) m = m * c.gamma1;
                        t[0] = m * c.kern.template w<KAHAN>(xk - xyz<R>(d.x));
                        return 1u;
                    });
    return group_total(acc, 0);
}

template <typename R, bool KAHAN>
__global__ void __launch_bounds__(kGroupThreads) k_group_sesph_density(int64_t n, State<R> s, Lists L,
                                                                       SolverConsts<R> c, const int* FSB_R status) {
    chain_entry();
    phase_begins(s.phase_at, 1);
    __shared__ GroupRows<R, 1> rows[kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const R r = group_density<R, KAHAN, true>(kk, fluid ? L.size(kk) : 0u, xyz<R>(s.pos[kk]), s, L, c,
                                              rows[threadIdx.x / kGroup]);
    if (!fluid || group_lane() != 0) return;
    s.rho[k] = r;
    const R pr = c.stiffness * (r / c.rest_density - R(1));
    s.p[k] = (pr < R(0)) ? R(0) : pr;
}

// the split first loop's density: 3D (IISPHFluidSolver3D) or 2D
template <typename R, bool KAHAN, bool GAMMA>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph_density(int64_t n, State<R> s, Lists L,
                                                                       SolverConsts<R> c, const int* FSB_R status) {
    phase_begins(s.phase_at, 1);
    __shared__ GroupRows<R, 1> rows[kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool in = k < n, fluid = in && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = in ? k : 0;
    const R r = group_density<R, KAHAN, GAMMA>(kk, fluid ? L.size(kk) : 0u, xyz<R>(s.pos[kk]), s, L, c,
                                               rows[threadIdx.x / kGroup]);
    if (in && group_lane() == 0) s.rho[k] = fluid ? r : s.rho_prev[k];
}

// ---------------------------------------------------------------------------
// SESPH accelerations (sesph_accel_one)
// ---------------------------------------------------------------------------
template <typename R, bool KAHAN>
__global__ void __launch_bounds__(kGroupThreads) k_group_sesph_accel(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                                     const int* FSB_R status) {
    chain_entry();
    phase_begins(s.phase_at, 2);
    __shared__ GroupRows<R, 6> rows[kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const V4<R> pk = s.pos[kk];
    const V3<R> xk = xyz<R>(pk), vk = xyz<R>(s.vel[kk]);
    const R rk = s.rho[kk];
    const R pdd = rk == R(0) ? R(0) : s.p[kk] / (rk * rk);
    Acc<R, KAHAN> acc;   // viscosity 0-2, pressure 3-5
    group_sum<6, 3>(L, kk, fluid ? L.size(kk) : 0u, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t) { return GForce<R>{s.pos[j], s.vel[j], s.rho[j], s.p[j]}; },
                    [&](uint32_t e, const GForce<R>& d, R* t) {
                        const V3<R> xij = xk - xyz<R>(d.x);
                        const V3<R> g = c.kern.template grad<KAHAN>(xij);
                        const bool visc = viscosity_term<R, KAHAN>(c, xij, g, vk - xyz<R>(d.v), d.x.w, d.rho, t);
                        V3<R> p;
                        if (e & kBoundaryBit) {
                            const R f = -pk.w * (pdd + pdd);
                            p = c.single_layer ? (f * g) * c.gamma2 : f * g;
                        } else {
                            const R pddj = d.rho == R(0) ? R(0) : fdiv<KAHAN>(d.p, d.rho * d.rho);
                            p = (-d.x.w * (pdd + pddj)) * g;
                        }
                        put3(t + 3, p);
                        return visc ? 3u : 2u;
                    });
    const V3<R> visc = group_total3(acc, 0), pa = group_total3(acc, 3);
    if (!fluid || group_lane() != 0) return;
    V3<R> npa = v3<R>(R(0), R(0), R(0)) + v3<R>(R(0), -c.gravity, R(0));
    npa = npa + c.two_nu * visc;
    s.acc[k] = v4<R>(pa + npa, R(0));
}

// ---------------------------------------------------------------------------
// IISPH first loop (iisph3d_l1_one, iisph2d_l1_at)
// ---------------------------------------------------------------------------
// Stores the gradients where the context keeps them (G.g not null).
// TWO_D: IISPHFluidSolver's loop (no pressure reset, no a_np; a particle's own
// density is the new one). SPLIT: the density has run before, and viscosity
// reads a fluid neighbor with a smaller host index at its new density.
template <typename R, bool KAHAN, bool SPLIT, bool TWO_D>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph_l1(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                                  Gradients<R> G, const StepScalars* FSB_R sc,
                                                                  const int* FSB_R status) {
    phase_begins(s.phase_at, 1);
    __shared__ GroupRows<R, 3> rows3[kGroupsPerBlock];
    __shared__ GroupRows<R, 1> rows1[SPLIT ? 1 : kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool in = k < n;
    const uint8_t ty = in ? s.type[k] : (uint8_t)FS_TYPE_INACTIVE;
    const bool fluid = ty == FS_TYPE_NORMAL;
    const int64_t kk = in ? k : 0;
    const V4<R> pk = s.pos[kk], vk = s.vel[kk];
    const uint32_t nn = fluid ? L.size(kk) : 0u;
    R rk = s.rho_prev[kk];
    if constexpr (!SPLIT) {
        const R r = group_density<R, KAHAN, !TWO_D>(kk, nn, xyz<R>(pk), s, L, c, rows1[threadIdx.x / kGroup]);
        if (fluid) rk = r;
    } else {
        rk = s.rho[kk];
    }
    const uint32_t hk = SPLIT ? s.hidx[kk] : 0u;
    Acc<R, KAHAN> acc;
    group_sum<3, 3>(L, kk, nn, rows3[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                        R rj = s.rho_prev[j];
                        // (a boundary particle's density is the same in both)
                        if (SPLIT && s.hidx[j] < hk) rj = s.rho[j];
                        return GVisc<R>{s.pos[j], s.vel[j], rj, at};
                    },
                    [&](uint32_t e, const GVisc<R>& d, R* t) {
                        const V3<R> xij = xyz<R>(pk) - xyz<R>(d.x);
                        R rj = d.rho;
                        if (TWO_D && (e & kIndexMask) == (uint32_t)k) rj = rk;
                        const V3<R> g = c.kern.template grad<KAHAN>(xij);
                        if (G.g && d.at >= 0) G.g[d.at] = v4<R>(g, d.x.w);   // for the passes that follow
                        return viscosity_term<R, KAHAN>(c, xij, g, xyz<R>(vk) - xyz<R>(d.v), d.x.w, rj, t) ? 1u : 0u;
                    });
    const V3<R> visc = group_total3(acc, 0);
    if (!in || group_lane() != 0) return;
    if (ty == FS_TYPE_INACTIVE) {
        if (!SPLIT) s.rho[k] = s.rho_prev[k];   // carry the density through the double buffer
        return;
    }
    if (!TWO_D) s.p[k] = R(0);
    V3<R> npa = xyz<R>(s.ext[k]);
    if (ty != FS_TYPE_BOUNDARY) {
        npa = npa + v3<R>(R(0), -c.gravity, R(0));
        npa = npa + c.two_nu * visc;
    }
    s.vstar[k] = v4<R>(xyz<R>(vk) + (R)sc->dt * npa, R(0));
    if (!TWO_D) s.anp[k] = v4<R>(npa, R(0));
    s.ext[k] = v4<R>(v3<R>(R(0), R(0), R(0)), R(0));
    if (!SPLIT) s.rho[k] = rk;   // boundary: the previous density
}

// ---------------------------------------------------------------------------
// IISPH 3D second loop and pressure iteration (iisph3d_l2_one, ...)
// ---------------------------------------------------------------------------
template <typename R, bool KAHAN, bool TWO_PASS, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph3d_l2(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                                    Gradients<R> G,
                                                                    const StepScalars* FSB_R sc,
                                                                    const int* FSB_R status) {
    phase_begins(s.phase_at, 2);
    constexpr int NC = TWO_PASS ? 4 : 8;
    __shared__ GroupRows<R, NC> rows[kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const uint32_t nn = fluid ? L.size(kk) : 0u;
    const V4<R> pk = s.pos[kk], vsk4 = s.vstar[kk];
    const V3<R> xk = xyz<R>(pk), vsk = xyz<R>(vsk4);
    // contrib 0, inner 1-3; in the single pass sum m gradW 4-6 and sum_fluid m |gradW|^2 7
    Acc<R, KAHAN> acc;
    group_sum<NC, TWO_PASS ? NC : 7>(L, kk, nn, rows[threadIdx.x / kGroup], acc,
                                     [&](uint32_t j, int64_t at) {
                                         return GPosVec<R>{position_or_gradient<CACHED>(s, G, j, at), s.vstar[j]};
                                     },
                                     [&](uint32_t e, const GPosVec<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        const bool bnd = (e & kBoundaryBit) != 0u;
        V3<R> in;
        if (!bnd) {
            t[0] = d.x.w * dotf<KAHAN>(vsk - xyz<R>(d.v), g);
            in = (KAHAN ? d.x.w * c.inv_rho0_sq : d.x.w / c.rho0_sq) * g;
        } else {
            t[0] = d.x.w * dotf<KAHAN>(vsk, g);
            const R w = c.single_layer ? c.two_gamma * d.x.w : R(2) * d.x.w;
            in = (KAHAN ? w * c.inv_rho0_sq : w / c.rho0_sq) * g;
        }
        put3(t + 1, -in);
        if constexpr (!TWO_PASS) {
            put3(t + 4, d.x.w * g);
            t[7] = d.x.w * dotf<KAHAN>(g, g);
        }
        return bnd ? 1u : 3u;
    });
    const R contrib = group_total(acc, 0);
    const V3<R> in = group_total3(acc, 1);
    const R dt = (R)sc->dt;
    R diag;
    if constexpr (TWO_PASS) {
        __shared__ GroupRows<R, 2> rows2[kGroupsPerBlock];
        Acc<R, KAHAN> d;
        const R mi = pk.w / c.rho0_sq;
        group_sum<2, 1, true>(L, kk, nn, rows2[threadIdx.x / kGroup], d,
                              [&](uint32_t j, int64_t at) {
                                  return GPos<R>{position_or_gradient<CACHED>(s, G, j, at)};
                              },
                              [&](uint32_t e, const GPos<R>& q, R* t) {
            const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, q.x);
            t[0] = q.x.w * dot(in, g);
            t[1] = q.x.w * dot(mi * (-g), g);
            return (e & kBoundaryBit) ? 1u : 3u;
        });
        diag = group_total(d, 0) * (dt * dt);
    } else {
        const V3<R> mg = group_total3(acc, 4);
        const R mg2 = group_total(acc, 7);
        diag = (dot(in, mg) - (pk.w / c.rho0_sq) * mg2) * (dt * dt);
    }
    if (!fluid || group_lane() != 0) return;
    const R source = (c.rest_density - s.rho[k]) - dt * contrib;
    s.vstar[k] = v4<R>(vsk, source);
    s.anp[k].w = diag;
}

template <typename R, bool KAHAN, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph3d_pressure_acc(int64_t n, State<R> s, Lists L,
                                                                              SolverConsts<R> c, Gradients<R> G,
                                                                              const StepScalars* FSB_R sc,
                                                                              const int* FSB_R status) {
    phase_begins(s.phase_at, 3);
    __shared__ GroupRows<R, 3> rows[kGroupsPerBlock];
    if (*status || sc->done) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const V3<R> xk = xyz<R>(s.pos[kk]);
    const R pk = s.p[kk];
    const R qk = pk / c.rho0_sq;
    Acc<R, KAHAN> acc;
    group_sum<3, 3>(L, kk, fluid ? L.size(kk) : 0u, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                        return GPosScalar<R>{position_or_gradient<CACHED>(s, G, j, at), s.p[j]};
                    },
                    [&](uint32_t e, const GPosScalar<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        const bool bnd = (e & kBoundaryBit) != 0u;
        V3<R> v;
        if (KAHAN) {
            const R f = !bnd ? d.x.w * (pk + d.a) : (c.single_layer ? c.two_gamma : R(2)) * d.x.w * pk;
            v = (f * c.inv_rho0_sq) * g;
        } else if (!bnd) {
            v = (d.x.w * (qk + d.a / c.rho0_sq)) * g;
        } else if (c.single_layer) {
            v = ((((c.gamma * d.x.w) * R(2)) * pk) / c.rho0_sq) * g;
        } else {
            v = (((d.x.w * R(2)) * pk) / c.rho0_sq) * g;
        }
        put3(t, -v);
        return 1u;
    });
    const V3<R> a = group_total3(acc, 0);
    if (fluid && group_lane() == 0) s.acc[k] = v4<R>(a, R(0));
}

template <typename R, bool KAHAN, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph3d_pressure_update(int64_t n, State<R> s, Lists L,
                                                                                 SolverConsts<R> c, Gradients<R> G,
                                                                                 StepScalars* FSB_R sc,
                                                                                 const int* FSB_R status) {
    __shared__ GroupRows<R, 1> rows[kGroupsPerBlock];
    if (*status || sc->done) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const V3<R> xk = xyz<R>(s.pos[kk]), ak = xyz<R>(s.acc[kk]);
    Acc<R, KAHAN> acc;
    group_sum<1, 1>(L, kk, fluid ? L.size(kk) : 0u, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                        return GPosVec<R>{position_or_gradient<CACHED>(s, G, j, at), s.acc[j]};
                    },
                    [&](uint32_t e, const GPosVec<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        t[0] = d.x.w * ((e & kBoundaryBit) ? dotf<KAHAN>(ak, g) : dotf<KAHAN>(ak - xyz<R>(d.v), g));
        return 1u;
    });
    const R ap = group_total(acc, 0);
    ErrPart o;
    if (fluid && group_lane() == 0)
        o = iisph3d_pressure_update_tail<R>(k, s, c, (R)sc->dt, ak, ap, s.vstar[k], s.anp[k].w, s.p[k]);
    reduce_err_parts(o, sc);
}

// ---------------------------------------------------------------------------
// IISPH 2D second loop and pressure iteration (iisph2d_l2_at, ...)
// ---------------------------------------------------------------------------
template <typename R, bool KAHAN, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph2d_l2(int64_t n, State<R> s, Lists L, SolverConsts<R> c,
                                                                    Gradients<R> G,
                                                                    const StepScalars* FSB_R sc,
                                                                    const int* FSB_R status) {
    phase_begins(s.phase_at, 2);
    __shared__ GroupRows<R, 4> rows[kGroupsPerBlock];
    __shared__ GroupRows<R, 1> rows1[kGroupsPerBlock];
    if (*status) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const uint32_t nn = fluid ? L.size(kk) : 0u;
    const V4<R> pk = s.pos[kk];
    const V3<R> xk = xyz<R>(pk), vsk = xyz<R>(s.vstar[kk]);
    Acc<R, KAHAN> acc;   // sum 0, internal 1-3
    group_sum<4, 4>(L, kk, nn, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                                         return GPosVec<R>{position_or_gradient<CACHED>(s, G, j, at), s.vstar[j]};
                                     },
                    [&](uint32_t e, const GPosVec<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        t[0] = d.x.w * dot(vsk - xyz<R>(d.v), g);
        if (!(e & kBoundaryBit)) put3(t + 1, ((d.x.w / c.rest_density) / c.rest_density) * g);
        else put3(t + 1, (((c.two_gamma * d.x.w) / c.rest_density) / c.rest_density) * g);
        return 1u;
    });
    const R sum = group_total(acc, 0);
    const V3<R> neg_in = -group_total3(acc, 1);
    const R mi = (pk.w / c.rest_density) / c.rest_density;
    auto pos = [&](uint32_t j, int64_t at) { return GPos<R>{position_or_gradient<CACHED>(s, G, j, at)}; };
    GroupRows<R, 1>& row = rows1[threadIdx.x / kGroup];
    Acc<R, KAHAN> d;   // over every neighbor, then over the fluid ones
    group_sum<1, 1>(L, kk, nn, row, d, pos, [&](uint32_t, const GPos<R>& q, R* t) {
        t[0] = q.x.w * dot(neg_in, gradient_of<CACHED, KAHAN>(c, xk, q.x));
        return 1u;
    });
    group_sum<1, 1>(L, kk, nn, row, d, pos, [&](uint32_t e, const GPos<R>& q, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, q.x);
        t[0] = q.x.w * dot(mi * (-g), g);
        return (e & kBoundaryBit) ? 0u : 1u;
    });
    const R dd = group_total(d, 0);
    if (!fluid || group_lane() != 0) return;
    const R dt = (R)sc->dt;
    const R source = (c.rest_density - s.rho[k]) - dt * sum;
    s.vstar[k] = v4<R>(vsk, source);
    s.anp[k] = v4<R>(v3<R>(R(0), R(0), R(0)), (dt * dt) * dd);
    s.p[k] = R(0);
}

template <typename R, bool KAHAN, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph2d_pressure_acc(int64_t n, State<R> s, Lists L,
                                                                              SolverConsts<R> c, Gradients<R> G,
                                                                              const StepScalars* FSB_R sc,
                                                                              const int* FSB_R status) {
    phase_begins(s.phase_at, 3);
    __shared__ GroupRows<R, 3> rows[kGroupsPerBlock];
    if (*status || sc->done) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const V3<R> xk = xyz<R>(s.pos[kk]);
    const R pr = (s.p[kk] / c.rest_density) / c.rest_density;
    Acc<R, KAHAN> acc;
    group_sum<3, 3>(L, kk, fluid ? L.size(kk) : 0u, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                        return GPosScalar<R>{position_or_gradient<CACHED>(s, G, j, at), s.p[j]};
                    },
                    [&](uint32_t e, const GPosScalar<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        if (!(e & kBoundaryBit)) put3(t, (d.x.w * (pr + (d.a / c.rest_density) / c.rest_density)) * g);
        else put3(t, (((c.gamma * d.x.w) * R(2)) * pr) * g);
        return 1u;
    });
    const V3<R> a = group_total3(acc, 0);
    if (fluid && group_lane() == 0) s.acc[k] = v4<R>(-a, R(0));
}

template <typename R, bool KAHAN, bool CACHED>
__global__ void __launch_bounds__(kGroupThreads) k_group_iisph2d_pressure_update(int64_t n, State<R> s, Lists L,
                                                                                 SolverConsts<R> c, Gradients<R> G,
                                                                                 StepScalars* FSB_R sc,
                                                                                 const int* FSB_R status) {
    __shared__ GroupRows<R, 1> rows[kGroupsPerBlock];
    if (*status || sc->done) return;
    const int64_t k = group_owner();
    const bool fluid = k < n && s.type[k] == FS_TYPE_NORMAL;
    const int64_t kk = fluid ? k : 0;
    const V3<R> xk = xyz<R>(s.pos[kk]), ak = xyz<R>(s.acc[kk]);
    Acc<R, KAHAN> acc;
    group_sum<1, 1>(L, kk, fluid ? L.size(kk) : 0u, rows[threadIdx.x / kGroup], acc,
                    [&](uint32_t j, int64_t at) {
                        return GPosVec<R>{position_or_gradient<CACHED>(s, G, j, at), s.acc[j]};
                    },
                    [&](uint32_t e, const GPosVec<R>& d, R* t) {
        const V3<R> g = gradient_of<CACHED, KAHAN>(c, xk, d.x);
        t[0] = d.x.w * ((e & kBoundaryBit) ? dot(ak, g) : dot(ak - xyz<R>(d.v), g));
        return 1u;
    });
    const R sum = group_total(acc, 0);
    double e_sum = 0.0;
    unsigned int e_cnt = 0;
    if (fluid && group_lane() == 0) iisph2d_pressure_update_tail<R>(k, s, c, (R)sc->dt, sum, e_sum, e_cnt);
    e_sum = warp_sum(e_sum);
    e_cnt = warp_sum(e_cnt);
    if ((threadIdx.x & 31) == 0 && e_cnt) {
        atomicAdd(&sc->err_sum, e_sum);
        atomicAdd(&sc->err_count, (unsigned long long)e_cnt);
    }
}

// ---------------------------------------------------------------------------
// solver lists with kGroup threads per owner
// ---------------------------------------------------------------------------
// The lists of k_build_lists (and, SORT, k_sort_lists_by_host), entry for entry.
// The group's threads look up the ranges of sorted particles that the walk
// visits (a cell and region each, or rows of three cells away from the grid's
// border), all together; list their particles in the walk's order; and test
// them kGroup at a time, the hits taking their places by ballot. SORT: a hit's
// place is the number of hits with a smaller host index. Owners whose
// neighborhood leaves the grid take the serial walk, which checks every
// candidate's own cell. ROUNDS: ranges per thread, 18 in 2D and at most 54 in
// 3D over kGroup.
//
// One thread per owner walks 9 or 27 cells in a row: 28 us for the 3,688
// particles of a 2D dam. fs_api.cu (grouped_lists) has the sizes at which each
// is faster, and the times.
constexpr int kListWindow = 128;   // candidates listed at a time; hits sorted in shared memory
struct ListGroup {
    uint32_t cand[kListWindow];
};
struct ListSort {
    uint32_t hit[kListWindow], host[kListWindow];
};
template <typename R, int ROUNDS, bool SORT>
__global__ void __launch_bounds__(kGroupThreads) k_group_lists(int64_t n_owners, const V4<R>* FSB_R pos,
                                                               const uint8_t* FSB_R type, const uint32_t* FSB_R hidx,
                                                               const uint32_t* FSB_R cell_start, WalkParams w,
                                                               uint32_t owner_mask, bool rows, uint32_t* FSB_R nbr,
                                                               int64_t stride, int K, uint32_t* FSB_R count,
                                                               int* FSB_R status, StepScalars* FSB_R sc) {
    chain_entry();
    __shared__ ListGroup lists[kGroupsPerBlock];
    __shared__ ListSort sorts[SORT ? kGroupsPerBlock : 1];
    {   // an overflow elsewhere does not stop the counting: the largest list decides how far the lists grow
        const int err = *status;
        if (err && err != FS_ERR_CAPACITY) return;
    }
    const unsigned all = 0xffffffffu, shift = threadIdx.x & 31u & ~(unsigned)(kGroup - 1);
    constexpr unsigned kMask = (1u << kGroup) - 1u;
    const int g = group_lane();
    ListGroup& sh = lists[threadIdx.x / kGroup];
    const int64_t k = group_owner();
    const bool in = k < n_owners;
    const int64_t kk = in ? k : 0;
    const bool owner = in && ((owner_mask >> type[kk]) & 1u);
    const V3<R> xi = xyz<R>(pos[kk]);
    const SceneGrid gr = w.grid_of(kk);
    const int c0 = cell_coord<R>(xi.x, w.r, w.trunc), c1 = cell_coord<R>(xi.y, w.r, w.trunc),
              c2 = cell_coord<R>(xi.z, w.r, w.trunc);
    const int l0 = c0 - gr.o0, l1 = c1 - gr.o1, l2 = c2 - gr.o2;
    // walk_rows' condition, and whether every neighbor cell lies in the grid
    const bool row = rows && !(l0 < 2 || l1 < 2 || l2 < 2 || l0 > gr.d0 - 3 || l1 > gr.d1 - 3 || l2 > gr.d2 - 3);
    const bool inside = l0 >= 1 && l1 >= 1 && l0 < gr.d0 - 1 && l1 < gr.d1 - 1 &&
                        (w.dim == 2 ? l2 >= 0 && l2 < gr.d2 : l2 >= 1 && l2 < gr.d2 - 1);
    const int nranges = !owner || !inside ? 0 : row ? 18 : (w.dim == 2 ? 9 : 27) * w.regions;
    uint32_t rb[ROUNDS], rn[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int q = r * kGroup + g;
        rb[r] = rn[r] = 0u;
        if (q >= nranges) continue;
        int region, x, y, z, len = 1;
        if (row) {
            region = q / 9;
            x = l0 - 1;
            y = l1 + q % 9 % 3 - 1;
            z = l2 + q % 9 / 3 - 1;
            len = 3;
        } else {   // cells dx, dy, dz ascending, the regions of a cell together
            const int c = w.regions == 2 ? q >> 1 : q;
            region = w.regions == 2 ? q & 1 : 0;
            x = l0 + (w.dim == 2 ? c / 3 : c / 9) - 1;
            y = l1 + (w.dim == 2 ? c % 3 : c / 3 % 3) - 1;
            z = l2 + (w.dim == 2 ? 0 : c % 3 - 1);
        }
        const uint32_t* cs = cell_start + region * (w.cells + 1) + gr.base + ((int64_t)z * gr.d1 + y) * gr.d0 + x;
        rb[r] = cs[0] | (region == 1 ? kBoundaryBit : 0u);
        rn[r] = cs[len] - cs[0];
    }
    // places of the ranges in the list of candidates
    uint32_t off[ROUNDS], total = 0;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        uint32_t incl = rn[r];
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) {
            const uint32_t y = __shfl_up_sync(all, incl, o, kGroup);
            if (g >= o) incl += y;
        }
        off[r] = total + incl - rn[r];
        total += __shfl_sync(all, incl, kGroup - 1, kGroup);
    }
    const uint32_t most = __reduce_max_sync(all, total);
    const float x0 = (float)xi.x, x1 = (float)xi.y, x2 = (float)xi.z;
    uint32_t c = 0;
    for (uint32_t base = 0; base < most; base += kListWindow) {
#pragma unroll
        for (int r = 0; r < ROUNDS; r++) {
            const uint32_t to = min(off[r] + rn[r], base + kListWindow);
            for (uint32_t i = max(off[r], base); i < to; i++) sh.cand[i - base] = rb[r] + (i - off[r]);
        }
        __syncwarp();
        const uint32_t m = total > base ? min(total - base, (uint32_t)kListWindow) : 0u;
        const uint32_t mm = __reduce_max_sync(all, m);
        constexpr int U = 4;   // candidates in flight per thread
        for (uint32_t i = 0; i < mm; i += kGroup * U) {
            uint32_t j[U];
            V4<R> pj[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t q = i + u * kGroup + g;
                j[u] = q < m ? sh.cand[q] : 0u;
                pj[u] = pos[j[u] & kIndexMask];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                bool hit = i + u * kGroup + g < m;
                if (row) {
                    const float d0 = x0 - (float)pj[u].x, d1 = x1 - (float)pj[u].y, d2 = x2 - (float)pj[u].z;
                    hit = hit && (d0 * d0 + d1 * d1) + d2 * d2 <= w.r2;
                } else {
                    hit = hit && within<R>(xi - xyz<R>(pj[u]), w);
                }
                uint32_t e = j[u];
                if (hit && w.regions == 1) {   // one region for all types
                    const uint8_t tj = type[e];
                    hit = tj != FS_TYPE_INACTIVE;
                    if (tj == FS_TYPE_BOUNDARY) e |= kBoundaryBit;
                }
                const unsigned bal = (__ballot_sync(all, hit) >> shift) & kMask;
                const uint32_t at = c + __popc(bal & ((1u << g) - 1u));
                if (hit) {
                    if (SORT && at < (uint32_t)kListWindow) {
                        sorts[threadIdx.x / kGroup].hit[at] = e;
                        sorts[threadIdx.x / kGroup].host[at] = hidx[e & kIndexMask];
                    } else if ((int)at < K) {
                        nbr[(int64_t)at * stride + k] = e;
                    }
                }
                c += __popc(bal);
            }
        }
        __syncwarp();
    }
    if (SORT && c > 0) {
        ListSort& so = sorts[threadIdx.x / kGroup];
        const int h = (int)min(c, (uint32_t)kListWindow);
        for (int a = g; a < h; a += kGroup) {
            const uint32_t mine = so.host[a];
            int place = a;
            if (c <= (uint32_t)kListWindow) {
                place = 0;
                for (int b = 0; b < h; b++) place += so.host[b] < mine ? 1 : 0;
            }
            if (place < K) nbr[(int64_t)place * stride + k] = so.hit[a];
        }
    }
    // the block's first threads, one per owner, note the lengths and walk for the
    // owners whose neighborhood leaves the grid: side by side in one warp, for a
    // lane in each of four warps took 2.6 ms where that takes 1.9 (a step of 2,000
    // particles in the border of a clamped grid)
    __shared__ uint32_t lengths[kGroupsPerBlock];
    constexpr uint32_t kWalk = 0xffffffffu;
    if (g == 0) lengths[threadIdx.x / kGroup] = owner && !inside ? kWalk : c;
    __syncthreads();
    if (threadIdx.x < kGroupsPerBlock) {
        const int64_t o = blockIdx.x * (int64_t)kGroupsPerBlock + threadIdx.x;
        if (o < n_owners) {
            uint32_t m = lengths[threadIdx.x];
            const bool walk = m == kWalk;
            if (walk) m = build_list_one<R>(o, pos, type, cell_start, w, rows, nbr, stride, K);
            count[o] = m;
            if (SORT && (m > (uint32_t)kListWindow || walk)) sort_list_by_host_at(o, nbr, stride, K, count, hidx);
            note_list_length(m, K, status, sc);
        }
    }
}

}  // namespace fsb
