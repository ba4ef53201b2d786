// The fluid path tracer of libFluid's visualizer (visualizer/raytracer/) on
// the device state: rays marched through the SPH density of the particles
// (ParticleIntersectionAccelerator.cpp), a stochastic path tracer over the
// surfaces they find (FluidRaytracer3D.cpp:70-200) with a white sky (the
// Skybox without an image, Skybox.cpp:27-31), and the pinhole camera of
// Camera.cpp:10-39. One warp per ray (fs_trace_rays) or per pixel (fs_render).
//
// A ray is a serial chain of march points, and an image of ordinary size has
// too few rays to hide the latency of a 27-cell walk per point behind one
// thread each: a 160 x 120 image is 600 warps of such threads, four per SM.
// So the lanes of a warp share a ray. They look at 32 march points at once
// for the next one with any particle in its 27 cells (a map with one byte per
// cell, k_neighborhood_map), and evaluate up to four points together: the
// candidates of all four are listed once and tested 32 at a time. The sums
// keep the walk's order (cells, regions, sorted order), so every density and
// normal is the same bit for bit as a serial walk's, and so is every path: the
// hits are compacted in order, the lanes evaluate the kernel for them in
// parallel, and one lane per sum adds its terms one by one. The normals,
// needed only where the surface is crossed, are evaluated there for the two
// points involved. Measured on a B200 (a 30 x 40 x 30 dam in its tank, 160 x
// 120, 1 sample, depth 10, the whole fs_render call): 26.6-37 ms with a thread
// per pixel, 2.8-3.3 ms now; the kernel issues on 42 % of cycles (399 M warp
// instructions for the camera rays alone, which cross many points near the
// walls) and is bound by its chains' fixed latencies. 24 instead of 16 warps
// per SM (80 registers) was slower, as was a second warp per pixel for the
// sky samples.
#pragma once

#include "fs_common.cuh"
#include "fs_search.cuh"
#include "fs_solvers.cuh"

namespace fsb {

struct RenderScene {
    float box_min[3], box_max[3];   // the particles' box, extended by the kernel support
    float step;                     // the march step, particle_size / 2
    float iso;                      // surface density: fraction * rest density
    SplineKernel<float> kern;
    WalkParams w;
    const uint8_t* map;             // per cell: whether its 27 cells hold any particle
};

__device__ __forceinline__ V3<float> lerp3(V3<float> a, V3<float> b, float f) {
    return v3<float>((1.0f - f) * a.x + b.x * f, (1.0f - f) * a.y + b.y * f, (1.0f - f) * a.z + b.z * f);
}

// Math::safe_normalize (LibFluidMath.hpp:36-42): zero where normalize gives NaN
__device__ __forceinline__ V3<float> safe_normalize(V3<float> v) {
    const float l = sqrtf(dot(v, v));
    const V3<float> r = v3<float>(v.x / l, v.y / l, v.z / l);
    if (isnan(r.x) || isnan(r.y) || isnan(r.z)) return v3<float>(0.f, 0.f, 0.f);
    return r;
}

// The volume at a march point without its normals.
struct VolumePoint {
    float density, fluid_density, boundary_density;
    V3<float> position;
};

// A warp evaluates up to kRayPoints march points of its ray together.
// Successive points lie half a particle size apart, so their 27-cell
// neighborhoods share most cells, and a walk's order -- cells by ascending x,
// then y, then z -- is the same for all of them: one list of the candidates of
// the union of the cells, in that order, serves every point, and a candidate
// outside a point's own 27 cells fails its distance test (at the radius
// itself, where rounding could let one pass, its kernel terms are below 1e-13
// of a particle's and leave the sums as they are).
constexpr int kRayPoints = 4;
constexpr int kRayWindow = 128;           // candidates listed at a time
constexpr int kRayRow = kRayWindow + 4;   // terms of a point's hits, padded to fours
constexpr int kRaySums = 12;              // 4 points x 3 densities, or 2 points x 6 normal components
struct alignas(16) RayShared {
    float term[kRaySums][kRayRow];
    uint32_t cand[kRayWindow];                // sorted index | kBoundaryBit in the boundary region
    uint32_t hit_a[kRayPoints][kRayWindow];   // densities: the squared distance's bits | kBoundaryBit (its sign)
    uint32_t hit_b[kRayPoints][kRayWindow];   // densities: the mass; normals: sorted index | kBoundaryBit
    float4 point[kRayPoints];
    float sum[kRaySums];
};
constexpr int kRayWarps = 4;   // rays per block (fs_trace_rays)

// enters particle j within the radius of x as hit `at` of point p
template <typename R, bool NORMALS>
__device__ __forceinline__ void put_hit(RayShared& sh, int p, int at, uint32_t j, bool bd, V3<float> x,
                                        const V4<R>& pj) {
    if (!NORMALS) {
        const V3<float> d = v3<float>(x.x - (float)pj.x, x.y - (float)pj.y, x.z - (float)pj.z);
        sh.hit_a[p][at] = __float_as_uint(dot(d, d)) | (bd ? kBoundaryBit : 0u);
        sh.hit_b[p][at] = __float_as_uint((float)pj.w);
    } else {
        sh.hit_b[p][at] = j | (bd ? kBoundaryBit : 0u);
    }
}

// Adds the terms of h0 .. h3 hits of the points 0 .. 3 to sh.sum, each sum's
// terms in order: the lanes evaluate the terms of all hits, then lane N p + i
// adds those of sum i of point p.
template <typename R, bool NORMALS>
__device__ __noinline__ void add_hits(int h0, int h1, int h2, int h3, const State<R>& s, const RenderScene& rs,
                                      RayShared& sh) {
    constexpr int N = NORMALS ? 6 : 3;
    const int lane = threadIdx.x & 31;
    // |d| / h: a multiplication where 1 / h is exact (h a power of two)
    const bool exact_inv = rs.kern.h * rs.kern.inv_h == 1.0f && (__float_as_uint(rs.kern.h) & 0x7fffffu) == 0;
    const int o1 = h0, o2 = o1 + h1, o3 = o2 + h2, total = o3 + h3;
    __syncwarp();
    for (int e = lane; e < total; e += 32) {
        const int p = (e >= o1) + (e >= o2) + (e >= o3);
        const int at = e - (p == 0 ? 0 : p == 1 ? o1 : p == 2 ? o2 : o3);
        float* row = &sh.term[N * p][at];
        const uint32_t hb = sh.hit_b[p][at];
        // the other type's sums get +0, which leaves them as they are
        if (!NORMALS) {
            const uint32_t ha = sh.hit_a[p][at];
            const bool bd = (ha & kBoundaryBit) != 0u;
            const float len = __fsqrt_rn(__uint_as_float(ha & kIndexMask));
            const float c = __uint_as_float(hb) * rs.kern.W_of(exact_inv ? len * rs.kern.inv_h : len / rs.kern.h);
            row[0] = c;
            row[kRayRow] = bd ? 0.f : c;
            row[2 * kRayRow] = bd ? c : 0.f;
        } else {
            const bool bd = (hb & kBoundaryBit) != 0u;
            const float4 x = sh.point[p];
            const V4<R> pj = s.pos[hb & kIndexMask];
            const V3<float> d = v3<float>(x.x - (float)pj.x, x.y - (float)pj.y, x.z - (float)pj.z);
            const float m = (float)pj.w;
            const V3<float> g = rs.kern.gradW(d);   // -GetKernelDerivativeValue(d)
            const float t[3] = {-(m * g.x), -(m * g.y), -(m * g.z)};
#pragma unroll
            for (int i = 0; i < 3; i++) {
                row[i * kRayRow] = bd ? 0.f : t[i];
                row[(3 + i) * kRayRow] = bd ? t[i] : 0.f;
            }
        }
    }
    if (lane < 16) {   // zeros up to a multiple of four
        const int p = lane >> 2, at = (p == 0 ? h0 : p == 1 ? h1 : p == 2 ? h2 : h3) + (lane & 3);
        if (N * p < kRaySums)
            for (int i = 0; i < N; i++) sh.term[N * p + i][at] = 0.f;
    }
    __syncwarp();
    if (lane < kRaySums) {
        const int p = lane / N, m = p == 0 ? h0 : p == 1 ? h1 : p == 2 ? h2 : h3;
        const float* row = sh.term[lane];
        float acc = sh.sum[lane];
        for (int h = 0; h < m; h += 4) {
            const float4 v = *reinterpret_cast<const float4*>(row + h);
            acc += v.x;
            acc += v.y;
            acc += v.z;
            acc += v.w;
        }
        sh.sum[lane] = acc;
    }
    __syncwarp();
}

// The serial walk of every point, which checks each particle's own cell: for
// points far apart, or at the border of a grid smaller than the particles'
// box, whose border cells hold clamped particles.
template <typename R, bool NORMALS>
__device__ __noinline__ void warp_sums_serial(int np, const State<R>& s, const uint32_t* __restrict__ cell_start,
                                              const RenderScene& rs, RayShared& sh) {
    for (int p = 0; p < np; p++) {
        const float4 q = sh.point[p];
        const V3<float> x = v3<float>(q.x, q.y, q.z);
        int at = 0;
        auto flush = [&] {
            add_hits<R, NORMALS>(p == 0 ? at : 0, p == 1 ? at : 0, p == 2 ? at : 0, p == 3 ? at : 0, s, rs, sh);
            at = 0;
        };
        walk_cells<R>(v3<R>((R)x.x, (R)x.y, (R)x.z), s.pos, s.type, cell_start, rs.w.grid_of(0), rs.w,
                      [&](uint32_t j, uint8_t tj) {
                          if (tj == FS_TYPE_INACTIVE) return;
                          put_hit<R, NORMALS>(sh, p, at, j, tj == FS_TYPE_BOUNDARY, x, s.pos[j]);   // every lane alike
                          if (++at == kRayWindow) flush();
                      });
        flush();
    }
}

// evaluate_volume_at_position (:76-126) for the points sh.point[0 .. np) by
// one warp: sums over the non-inactive particles within the search radius.
// NORMALS false: sh.sum[3 p ..] = density, fluid density and boundary density
// of point p; true (np <= 2): sh.sum[6 p ..] = the fluid and the boundary
// normal, sums of m_j GetKernelDerivativeValue(x - x_j).
template <typename R, bool NORMALS>
__device__ __noinline__ void warp_sums(int np, const State<R>& s, const uint32_t* __restrict__ cell_start,
                                       const RenderScene& rs, RayShared& sh) {
    constexpr int P = NORMALS ? 2 : kRayPoints;
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const WalkParams& w = rs.w;
    const SceneGrid gr = w.grid_of(0);
    if (lane < kRaySums) sh.sum[lane] = 0.f;
    V3<float> pt[P];
#pragma unroll
    for (int p = 0; p < P; p++) {
        const float4 q = sh.point[min(p, np - 1)];
        pt[p] = v3<float>(q.x, q.y, q.z);
    }
    // the union of the points' 27 cells: a box of at most 4 cells an axis, two
    // cells per lane in the walk's order (lane l: cells 2 l and 2 l + 1 of the
    // 4 x 4 x 4 box)
    const int org[3] = {gr.o0, gr.o1, gr.o2}, dim[3] = {gr.d0, gr.d1, gr.d2};
    int lo[3], ext[3];
    float bl[3], bh[3];   // the points' box, widened by the radius and a margin for the rounding of x / r
    bool simple = true;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        bl[a] = bh[a] = a == 0 ? pt[0].x : a == 1 ? pt[0].y : pt[0].z;
#pragma unroll
        for (int p = 1; p < P; p++) {
            const float c = a == 0 ? pt[p].x : a == 1 ? pt[p].y : pt[p].z;
            bl[a] = fminf(bl[a], c);
            bh[a] = fmaxf(bh[a], c);
        }
        // (cell coordinates ascend with positions: the box's corners hold the extreme cells)
        const int c0 = cell_coord<R>((R)bl[a], w.r, w.trunc), c1 = cell_coord<R>((R)bh[a], w.r, w.trunc);
        lo[a] = c0 - 1;
        ext[a] = c1 - c0 + 3;
        // within the grid, away from its border, and no more than 4 cells
        simple = simple && c1 >= c0 && c1 <= c0 + 1 && c0 > org[a] && c0 < org[a] + dim[a] && c1 < org[a] + dim[a] - 1;
        const float margin = 1e-3f * w.r + 1e-6f * (fabsf(bl[a]) + fabsf(bh[a]));
        bl[a] -= w.r + margin;   // a cell from `near` on holds no hit if near + r < bl + r or near > bh
        bh[a] += margin;
    }
    __syncwarp();
    if (!simple) {
        warp_sums_serial<R, NORMALS>(np, s, cell_start, rs, sh);
        return;
    }
    uint32_t rb[4] = {0, 0, 0, 0}, rn[4] = {0, 0, 0, 0};   // (cell, region) ranges in the walk's order
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int l = 2 * lane + q, x = l >> 4, y = (l >> 2) & 3, z = l & 3;
        if (x >= ext[0] || y >= ext[1] || z >= ext[2]) continue;
        const int c[3] = {lo[0] + x, lo[1] + y, lo[2] + z};
        // cells that lie farther from the points' box than the radius hold no hit
        float far2 = 0.f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float near = (float)c[a] * w.r;
            const float gap = fmaxf(fmaxf(near - bh[a], bl[a] - near), 0.f);
            far2 += gap * gap;
        }
        if (far2 > w.r2) continue;
        // (a grid has fewer than 2^30 cells)
        const uint32_t lc = ((uint32_t)(c[2] - org[2]) * (uint32_t)dim[1] + (uint32_t)(c[1] - org[1])) * (uint32_t)dim[0] +
                            (uint32_t)(c[0] - org[0]);
        rb[2 * q] = cell_start[lc];
        rn[2 * q] = cell_start[lc + 1] - rb[2 * q];
        if (w.regions > 1) {
            const uint32_t* cs = cell_start + (w.cells + 1);
            rb[2 * q + 1] = cs[lc];
            rn[2 * q + 1] = cs[lc + 1] - rb[2 * q + 1];
        }
    }
    const uint32_t own = rn[0] + rn[1] + rn[2] + rn[3];
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(all, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(all, incl, 31), first = incl - own;
    for (uint32_t base = 0; base < total; base += kRayWindow) {
        const uint32_t m = min(total - base, (uint32_t)kRayWindow);
        // this lane's candidates in the window
        uint32_t at = first;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t from = max(at, base), to = min(at + rn[q], base + m);
            const uint32_t flag = (q & 1) ? kBoundaryBit : 0u;
#pragma unroll 1
            for (uint32_t i = from; i < to; i++) sh.cand[i - base] = (rb[q] + (i - at)) | flag;
            at += rn[q];
        }
        __syncwarp();
        int hits[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (uint32_t i = 0; i < m; i += 32) {
            const uint32_t j = sh.cand[min(i + lane, m - 1)];
            const V4<R> pj = s.pos[j & kIndexMask];
            bool bd = (j & kBoundaryBit) != 0u, act = i + lane < m;
            if (w.regions == 1) {   // fluid and boundary in one region: the type tells
                const uint8_t tj = s.type[j];
                act = act && tj != FS_TYPE_INACTIVE;
                bd = tj == FS_TYPE_BOUNDARY;
            }
#pragma unroll
            for (int p = 0; p < P; p++) {
                const bool in = act && p < np &&
                                within<R>(v3<R>((R)pt[p].x, (R)pt[p].y, (R)pt[p].z) - xyz<R>(pj), w);
                const unsigned bal = __ballot_sync(all, in);
                if (in)
                    put_hit<R, NORMALS>(sh, p, hits[p] + __popc(bal & ((1u << lane) - 1u)), j & kIndexMask, bd, pt[p], pj);
                hits[p] += __popc(bal);
            }
        }
        add_hits<R, NORMALS>(hits[0], hits[1], hits[2], hits[3], s, rs, sh);
    }
}

// the interpolated normal of the crossing between last and cur: of the
// boundary's (type 2) or the fluid's density
template <typename R>
__device__ __forceinline__ V3<float> crossing_normal(const VolumePoint& last, const VolumePoint& cur, int type, float f,
                                                     const State<R>& s, const uint32_t* __restrict__ cell_start,
                                                     const RenderScene& rs, RayShared& sh) {
    __syncwarp();   // the densities in sh.sum have been read
    if ((threadIdx.x & 31) < 2) {
        const V3<float> x = (threadIdx.x & 31) == 0 ? last.position : cur.position;
        sh.point[threadIdx.x & 31] = make_float4(x.x, x.y, x.z, 0.f);
    }
    __syncwarp();
    warp_sums<R, true>(2, s, cell_start, rs, sh);
    const float* v = sh.sum + (type == 2 ? 3 : 0);
    const V3<float> n = safe_normalize(lerp3(v3<float>(v[0], v[1], v[2]), v3<float>(v[6], v[7], v[8]), f));
    __syncwarp();
    return n;
}

// map[c]: whether any particle of the structure lies in the 27 cells around
// cell c (set for the grid's outermost cells, whose neighborhood the grid
// does not hold)
static __global__ void k_neighborhood_map(const uint32_t* __restrict__ cell_start, WalkParams w,
                                          uint8_t* __restrict__ map) {
    const SceneGrid gr = w.grids[0];
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < w.cells;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % gr.d0), y = (int)(c / gr.d0 % gr.d1), z = (int)(c / gr.d0 / gr.d1);
        bool any = x < 1 || y < 1 || z < 1 || x > gr.d0 - 2 || y > gr.d1 - 2 || z > gr.d2 - 2;
        if (!any) {
            for (int g = 0; g < w.regions; g++) {
                const uint32_t* cs = cell_start + g * (w.cells + 1);
                for (int row = 0; row < 9; row++) {
                    const int64_t b = c + ((int64_t)(row / 3 - 1) * gr.d1 + (row % 3 - 1)) * gr.d0;
                    any = any || cs[b + 2] != cs[b - 1];
                }
            }
        }
        map[c] = any ? 1 : 0;
    }
}

// get_volume_state (:181-193): 0 outside, 1 fluid, 2 boundary
__device__ __forceinline__ int volume_state(const VolumePoint& e, float iso) {
    if (e.density < iso) return 0;
    return e.fluid_density > e.boundary_density ? 1 : 2;
}

// is_surface_intersected (:128-179). type: 0 the fluid surface reached from
// outside, 1 from inside, 2 a boundary surface; f: the crossing's place
// between the two points
__device__ __forceinline__ bool surface_crossed(const VolumePoint& last, const VolumePoint& cur, float iso, int& type,
                                                float& f) {
    const int ls = volume_state(last, iso), cs = volume_state(cur, iso);
    if (ls == cs || ls == 2) return false;
    if (ls == 0) {
        f = (iso - last.density) / (cur.density - last.density);
        type = cs == 1 ? 0 : 2;
    } else if (cs == 0) {
        f = (last.density - iso) / (last.density - cur.density);
        type = 1;
    } else {
        f = (last.boundary_density - last.fluid_density) /
            (cur.fluid_density - last.fluid_density - cur.boundary_density + last.boundary_density);
        type = 2;
    }
    return true;
}

// AABB::is_ray_intersecting (AABB.cpp:7-37), the slab test with Math::min/max
__device__ __forceinline__ bool box_hit(const RenderScene& rs, V3<float> o, V3<float> d) {
    const float tx1 = (rs.box_min[0] - o.x) / d.x, tx2 = (rs.box_max[0] - o.x) / d.x;
    const float txn = fminf(tx1, tx2), txf = fmaxf(tx1, tx2);
    const float ty1 = (rs.box_min[1] - o.y) / d.y, ty2 = (rs.box_max[1] - o.y) / d.y;
    const float tyn = fminf(ty1, ty2), tyf = fmaxf(ty1, ty2);
    if (txn > tyf || tyn > txf) return false;
    const float tn = fmaxf(txn, tyn), tf = fminf(txf, tyf);
    const float tz1 = (rs.box_min[2] - o.z) / d.z, tz2 = (rs.box_max[2] - o.z) / d.z;
    const float tzn = fminf(tz1, tz2), tzf = fmaxf(tz1, tz2);
    return !(tn > tzf || tzn > tf);
}

__device__ __forceinline__ bool box_contains(const RenderScene& rs, V3<float> p) {
    return !(p.x < rs.box_min[0] || p.x > rs.box_max[0] || p.y < rs.box_min[1] || p.y > rs.box_max[1] ||
             p.z < rs.box_min[2] || p.z > rs.box_max[2]);
}

// The t of a ray's march points that the box can hold (the slab range, widened
// by two steps); false where it holds none.
__device__ __forceinline__ bool march_range(V3<float> o, V3<float> d, float offset, const RenderScene& rs, long long& t0,
                                            long long& t1) {
    if (!box_hit(rs, o, d)) return false;
    constexpr long long kMaxSteps = 1000000;
    t0 = 1;
    t1 = kMaxSteps - 1;
    {
        float near = -INFINITY, far = INFINITY;
        const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
        bool ok = true;
        for (int a = 0; a < 3; a++) {
            const float u = (rs.box_min[a] - oo[a]) / dd[a], v = (rs.box_max[a] - oo[a]) / dd[a];
            if (isnan(u) || isnan(v)) ok = false;
            near = fmaxf(near, fminf(u, v));
            far = fminf(far, fmaxf(u, v));
        }
        if (ok) {
            if (far < 0.f) return false;   // the box lies behind the ray: every point is skipped
            const double lo = floor(((double)near - offset) / rs.step) - 2.0;
            const double hi = ceil(((double)far - offset) / rs.step) + 2.0;
            t0 = lo > 1.0 ? (long long)lo : 1;
            t1 = hi < (double)(kMaxSteps - 1) ? (long long)hi : kMaxSteps - 1;
        }
    }
    return true;
}

// whether any particle can lie in the 27 cells around p (a point whose cells the grid does not hold: it may)
template <typename R>
__device__ __forceinline__ bool occupied_around(V3<float> p, const SceneGrid& gr, const RenderScene& rs) {
    bool cl = false;
    const int l0 = local_cell(cell_coord<R>((R)p.x, rs.w.r, rs.w.trunc), gr.o0, gr.d0, cl);
    const int l1 = local_cell(cell_coord<R>((R)p.y, rs.w.r, rs.w.trunc), gr.o1, gr.d1, cl);
    const int l2 = local_cell(cell_coord<R>((R)p.z, rs.w.r, rs.w.trunc), gr.o2, gr.d2, cl);
    return cl || rs.map[gr.base + ((int64_t)l2 * gr.d1 + l1) * gr.d0 + l0] != 0;
}

// is_intersecting_with_particles (:20-74): march points x + (step t + offset) d,
// t = 1 .. 10^6 - 1, the surface is where the volume state changes. Points
// outside the box are skipped until the ray has entered it and end the march
// once it has left. Only the t whose points the box can hold are visited
// (march_range); the others would be skipped.
// Called by a whole warp for one ray: lane l looks at march point t + l, and
// the first point with particles around it, or the first past the box, is
// where the march goes on. Every point passed over has no particles in its 27
// cells: its densities are 0.
// want_normal false (occlusion): only whether there is a crossing counts.
template <typename R>
__device__ __noinline__ bool trace_ray(V3<float> o, V3<float> d, float offset, const State<R>& s,
                                       const uint32_t* __restrict__ cell_start, const RenderScene& rs, RayShared& sh,
                                       bool want_normal, int& type, V3<float>& point, V3<float>& normal,
                                       float& length) {
    long long t0, t1;
    if (!march_range(o, d, offset, rs, t0, t1)) return false;
    const int lane = threadIdx.x & 31;
    const SceneGrid gr = rs.w.grid_of(0);
    auto along = [&](float a) { return v3<float>(o.x + a * d.x, o.y + a * d.y, o.z + a * d.z); };
    auto at = [&](long long t) { return along(rs.step * (float)t + offset); };
    // the volume before the first march point, half a step along the ray
    VolumePoint last{0.f, 0.f, 0.f, along(rs.step / 2.0f)};
    bool have_last = false;
    // evaluates the volume at march points t .. t + np - 1 (np < kRayPoints until have_last:
    // last goes with them)
    auto evaluate = [&](long long t, int np) {
        const int extra = have_last ? 0 : 1;
        if (lane < np + extra) {
            const V3<float> x = lane < extra ? last.position : at(t + lane - extra);
            sh.point[lane] = make_float4(x.x, x.y, x.z, 0.f);
        }
        __syncwarp();
        warp_sums<R, false>(np + extra, s, cell_start, rs, sh);
        if (extra) last = VolumePoint{sh.sum[0], sh.sum[1], sh.sum[2], last.position};
        have_last = true;
        return extra;
    };
    auto cross = [&](const VolumePoint& cur, long long t) {
        float f;
        if (!surface_crossed(last, cur, rs.iso, type, f)) return false;
        point = lerp3(last.position, cur.position, f);
        length = rs.step * (float)t;
        if (want_normal) normal = crossing_normal<R>(last, cur, type, f, s, cell_start, rs, sh);
        return true;
    };
    bool within = false;
    for (long long t = t0; t <= t1; t += 32) {
        const long long mine = t + lane;
        bool in = false, full = false;
        if (mine <= t1) {
            const V3<float> p = at(mine);
            in = box_contains(rs, p);
            if (in) full = occupied_around<R>(p, gr, rs);
        }
        const unsigned inside = __ballot_sync(0xffffffffu, in), occupied = __ballot_sync(0xffffffffu, full);
        // points outside the box before the ray has entered it are passed over; the first one after it ends the march
        int pos = 0;
        if (!within) {
            if (!inside) continue;
            pos = __ffs(inside) - 1;
            within = true;
        }
        while (pos < 32) {
            if (!((inside >> pos) & 1u)) return false;   // past the box, or past t1
            if (!((occupied >> pos) & 1u)) {
                // a run of points with no particles around them: the densities are 0
                const unsigned rest = (occupied | ~inside) >> pos;
                const int end = rest ? pos + __ffs(rest) - 1 : 32;
                if (!have_last) {
                    evaluate(t + pos, 0);
                }
                const VolumePoint cur{0.f, 0.f, 0.f, at(t + pos)};
                if (cross(cur, t + pos)) return true;
                last = VolumePoint{0.f, 0.f, 0.f, at(t + end - 1)};
                pos = end;
                continue;
            }
            const unsigned run = ~(inside >> pos);   // points inside from here on
            const int ahead = min(run ? __ffs(run) - 1 : 32, 32 - pos);
            const int np = min(ahead, have_last ? kRayPoints : kRayPoints - 1);
            const int skip = evaluate(t + pos, np);
            VolumePoint cur[kRayPoints];
#pragma unroll
            for (int i = 0; i < kRayPoints; i++) {
                const float* v = sh.sum + 3 * min(i + skip, kRayPoints - 1);
                cur[i] = VolumePoint{v[0], v[1], v[2], at(t + pos + i)};
            }
#pragma unroll
            for (int i = 0; i < kRayPoints; i++) {
                if (i >= np) break;
                if (cross(cur[i], t + pos + i)) return true;
                last = cur[i];
            }
            __syncwarp();   // sh.sum has been read
            pos += np;
        }
    }
    return false;
}

__device__ __forceinline__ void store_hit(int64_t r, bool h, int type, V3<float> p, V3<float> n, float len,
                                          int32_t* __restrict__ hit, float* __restrict__ point,
                                          float* __restrict__ normal, float* __restrict__ length) {
    hit[r] = h ? type : -1;
    point[3 * r] = p.x;
    point[3 * r + 1] = p.y;
    point[3 * r + 2] = p.z;
    normal[3 * r] = n.x;
    normal[3 * r + 1] = n.y;
    normal[3 * r + 2] = n.z;
    length[r] = h ? len : -1.0f;
}

template <typename R>
__global__ void __launch_bounds__(32 * kRayWarps, 4) k_trace_rays(int64_t nrays, const float* __restrict__ origins, const float* __restrict__ dirs,
                             const __grid_constant__ State<R> s, const uint32_t* __restrict__ cell_start,
                             const __grid_constant__ RenderScene rs,
                             int32_t* __restrict__ hit, float* __restrict__ point, float* __restrict__ normal,
                             float* __restrict__ length) {
    __shared__ RayShared rays[kRayWarps];
    RayShared& sh = rays[threadIdx.x >> 5];
    const int64_t r = blockIdx.x * (int64_t)kRayWarps + (threadIdx.x >> 5);
    if (r >= nrays) return;
    const V3<float> o = v3<float>(origins[3 * r], origins[3 * r + 1], origins[3 * r + 2]);
    const V3<float> d = v3<float>(dirs[3 * r], dirs[3 * r + 1], dirs[3 * r + 2]);
    int type = -1;
    V3<float> p = v3<float>(0.f, 0.f, 0.f), n = p;
    float len = -1.0f;
    const bool h = trace_ray<R>(o, d, 0.0f, s, cell_start, rs, sh, true, type, p, n, len);
    if ((threadIdx.x & 31) == 0) store_hit(r, h, type, p, n, len, hit, point, normal, length);
}

// The same march by one thread, point by point: for many rays, whose number
// hides the latency of the chains. The sums are the walk's own, which the warp's
// equal bit for bit.
//
// B200, the whole fs_trace_rays call, a warp and a thread per ray: rays into a dam
// of 30,000 particles in its tank, 1,000 0.38 and 3.9 ms, 24,000 3.0 and 4.8, 32,000
// 3.7 and 4.9, 48,000 5.8 and 5.7, 64,000 7.2 and 6.1, 128,000 12.8 and 7.6; of
// 300,000, 32,000 4.0 and 6.6, 64,000 7.5 and 8.0, 128,000 13.4 and 9.4. (64 threads
// a block and the 72 registers that leaves it were faster than 128 of either from
// 96,000 on.)
constexpr int64_t kManyRays = 32768;   // rays up to which each has a warp
constexpr int kRayThreads = 64;
// NORMALS false: density, fluid density and boundary density at x; true: the
// fluid's or the boundary's normal.
template <typename R, bool NORMALS>
__device__ __forceinline__ void thread_sums(V3<float> x, bool boundary, const State<R>& s,
                                            const uint32_t* __restrict__ cell_start, const RenderScene& rs,
                                            float (&sum)[3]) {
    sum[0] = sum[1] = sum[2] = 0.f;
    walk_cells<R>(v3<R>((R)x.x, (R)x.y, (R)x.z), s.pos, s.type, cell_start, rs.w.grid_of(0), rs.w,
                  [&](uint32_t j, uint8_t tj) {
                      if (tj == FS_TYPE_INACTIVE) return;
                      const V4<R> pj = s.pos[j];
                      const V3<float> d = v3<float>(x.x - (float)pj.x, x.y - (float)pj.y, x.z - (float)pj.z);
                      const float m = (float)pj.w;
                      const bool bd = tj == FS_TYPE_BOUNDARY;
                      if (!NORMALS) {
                          const float c = m * rs.kern.W(d);
                          sum[0] += c;
                          if (bd) sum[2] += c;
                          else sum[1] += c;
                      } else {
                          const V3<float> g = rs.kern.gradW(d);   // -GetKernelDerivativeValue(d)
                          const V3<float> t = v3<float>(m * g.x, m * g.y, m * g.z);
                          if (bd == boundary) sum[0] -= t.x, sum[1] -= t.y, sum[2] -= t.z;
                      }
                  });
}
template <typename R>
__device__ bool thread_ray(V3<float> o, V3<float> d, const State<R>& s, const uint32_t* __restrict__ cell_start,
                           const RenderScene& rs, int& type, V3<float>& point, V3<float>& normal, float& length) {
    long long t0, t1;
    if (!march_range(o, d, 0.0f, rs, t0, t1)) return false;
    const SceneGrid gr = rs.w.grid_of(0);
    auto along = [&](float a) { return v3<float>(o.x + a * d.x, o.y + a * d.y, o.z + a * d.z); };
    auto at = [&](long long t) { return along(rs.step * (float)t + 0.0f); };
    auto volume = [&](V3<float> p, bool occupied) {
        float v[3] = {0.f, 0.f, 0.f};
        if (occupied) thread_sums<R, false>(p, false, s, cell_start, rs, v);
        return VolumePoint{v[0], v[1], v[2], p};
    };
    // the point before the first march point is evaluated as one of them
    VolumePoint last{0.f, 0.f, 0.f, along(rs.step / 2.0f)};
    bool have_last = false, within = false;
    V3<float> p = last.position;
    bool occupied = occupied_around<R>(p, gr, rs);
    for (long long t = t0; t <= t1;) {
        if (have_last && !box_contains(rs, p)) {
            if (within) break;
            p = at(++t);
            occupied = occupied_around<R>(p, gr, rs);
            continue;
        }
        // the next point's neighborhood, looked up under this one's sums
        const long long tn = have_last ? t + 1 : t;
        const V3<float> pn = at(tn);
        const bool next = occupied_around<R>(pn, gr, rs);
        const VolumePoint cur = volume(p, occupied);
        float f;
        if (have_last) {
            within = true;
            if (surface_crossed(last, cur, rs.iso, type, f)) {
                V3<float> n[2];
#pragma unroll 1
                for (int i = 0; i < 2; i++) {
                    float v[3];
                    thread_sums<R, true>(i == 0 ? last.position : cur.position, type == 2, s, cell_start, rs, v);
                    if (i == 0) n[0] = v3<float>(v[0], v[1], v[2]);
                    else n[1] = v3<float>(v[0], v[1], v[2]);
                }
                point = lerp3(last.position, cur.position, f);
                normal = safe_normalize(lerp3(n[0], n[1], f));
                length = rs.step * (float)t;
                return true;
            }
        }
        last = cur;
        have_last = true;
        t = tn;
        p = pn;
        occupied = next;
    }
    return false;
}
template <typename R>
__global__ void __launch_bounds__(kRayThreads) k_trace_many_rays(int64_t nrays, const float* __restrict__ origins,
                                                         const float* __restrict__ dirs,
                                                         const __grid_constant__ State<R> s,
                                                         const uint32_t* __restrict__ cell_start,
                                                         const __grid_constant__ RenderScene rs,
                                                         int32_t* __restrict__ hit, float* __restrict__ point,
                                                         float* __restrict__ normal, float* __restrict__ length) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nrays) return;
    int type = -1;
    V3<float> p = v3<float>(0.f, 0.f, 0.f), n = p;
    float len = -1.0f;
    const bool h = thread_ray<R>(v3<float>(origins[3 * r], origins[3 * r + 1], origins[3 * r + 2]),
                                 v3<float>(dirs[3 * r], dirs[3 * r + 1], dirs[3 * r + 2]), s, cell_start, rs, type, p, n, len);
    store_hit(r, h, type, p, n, len, hit, point, normal, length);
}

// the particles' box (calculate_aabb, :54-74), as ordered integer bits
__device__ __forceinline__ int ordered(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float unordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// (one atomic per warp and bound)
template <typename R>
__global__ void k_particle_box(int64_t n, State<R> s, int* __restrict__ box) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool in = k < n && s.type[k] != FS_TYPE_INACTIVE;
    V4<R> p{};
    if (in) p = s.pos[k];
    const float c[3] = {(float)p.x, (float)p.y, (float)p.z};
    for (int a = 0; a < 3; a++) {
        const int lo = __reduce_min_sync(0xffffffffu, in ? ordered(c[a]) : INT_MAX);
        const int hi = __reduce_max_sync(0xffffffffu, in ? ordered(c[a]) : INT_MIN);
        if ((threadIdx.x & 31) == 0) {
            if (lo != INT_MAX) atomicMin(&box[a], lo);
            if (hi != INT_MIN) atomicMax(&box[3 + a], hi);
        }
    }
}

// ---------------------------------------------------------------------------
// the path tracer (FluidRaytracer3D::evaluate_ray, :70-165)
// ---------------------------------------------------------------------------
struct RenderCamera {
    float pos[3];
    float right[3], up[3], back[3];   // the inverse view rotation's columns
    float tan_half_fov;
    int width, height, flip_y;
};
struct RenderShading {
    float fluid[3], boundary[3];      // bsdf: the colours (gamma 2.2 decoded) over pi
    int samples, max_depth, normals_only;
    unsigned long long seed;
};

// a counter-based stream of uniform floats in [0, 1) per pixel
struct PixelRng {
    unsigned long long key;
    unsigned int n = 0;
    __device__ float next() {
        unsigned long long z = key + 0x9E3779B97F4A7C15ull * (unsigned long long)(++n);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (float)(z >> 40) * (1.0f / 16777216.0f);
    }
};

// CosineWeightedHemisphereDistribution::sample_ray (CosineWeightedHemisphereDistribution.cpp:7-65)
__device__ void cosine_sample(float z1, float z2, V3<float> up, V3<float>& dir, float& solid_angle) {
    const float pi = 3.14159265358979323846f;
    const float x = cosf(2.0f * pi * z2) * sqrtf(z1), y = sinf(2.0f * pi * z2) * sqrtf(z1), z = sqrtf(1.0f - z1);
    V3<float> t;
    if (fabsf(up.x) > kFltEps) t = v3<float>((-up.y - up.z) / up.x, 1.0f, 1.0f);
    else if (fabsf(up.y) > kFltEps) t = v3<float>(1.0f, (-up.x - up.z) / up.y, 1.0f);
    else t = v3<float>(1.0f, 1.0f, (-up.x - up.y) / up.z);
    const float tl = sqrtf(dot(t, t));
    t = v3<float>(t.x / tl, t.y / tl, t.z / tl);
    V3<float> b = v3<float>(up.y * t.z - up.z * t.y, up.z * t.x - up.x * t.z, up.x * t.y - up.y * t.x);
    const float bl = sqrtf(dot(b, b));
    b = v3<float>(b.x / bl, b.y / bl, b.z / bl);
    dir = v3<float>(t.x * x + b.x * y + up.x * z, t.y * x + b.y * y + up.y * z, t.z * x + b.z * y + up.z * z);
    const float probability = cosf(asinf(sqrtf(z1))) / pi;
    solid_angle = 1.0f / probability;
}

template <typename R>
__global__ void __launch_bounds__(32 * kRayWarps, 4) k_render(const __grid_constant__ State<R> s,
                                                                const uint32_t* __restrict__ cell_start,
                                                                const __grid_constant__ RenderScene rs,
                                                                const __grid_constant__ RenderCamera cam,
                                                                const __grid_constant__ RenderShading sh,
                                                                float* __restrict__ radiance) {
    __shared__ RayShared rays[kRayWarps];
    RayShared& sh_ray = rays[threadIdx.x >> 5];
    const int px = blockIdx.x * kRayWarps + (threadIdx.x >> 5);   // the warp's pixel: every lane follows its path
    const int w = cam.width, h = cam.height;
    if (px >= w * h) return;
    const int x = px % w, y = px / w;
    PixelRng rng{sh.seed ^ (0xD1B54A32D192ED03ull * (unsigned long long)(px + 1))};
    // Camera::generate_ray_for_sample_position (Camera.cpp:10-39); its aspect ratio is width / width
    float rx = ((float)x + 0.5f) / (float)w * 2.0f - 1.0f, ry = ((float)y + 0.5f) / (float)h * 2.0f - 1.0f;
    if (!cam.flip_y) ry = -ry;
    V3<float> pv = v3<float>(rx * cam.tan_half_fov, ry * cam.tan_half_fov, -1.0f);
    const float pl = sqrtf(dot(pv, pv));
    pv = v3<float>(pv.x / pl, pv.y / pl, pv.z / pl);
    V3<float> dir = v3<float>(cam.right[0] * pv.x + cam.up[0] * pv.y + cam.back[0] * pv.z,
                              cam.right[1] * pv.x + cam.up[1] * pv.y + cam.back[1] * pv.z,
                              cam.right[2] * pv.x + cam.up[2] * pv.y + cam.back[2] * pv.z);
    const float dl = sqrtf(dot(dir, dir));
    dir = v3<float>(dir.x / dl, dir.y / dl, dir.z / dl);
    const V3<float> origin = v3<float>(cam.pos[0], cam.pos[1], cam.pos[2]);
    auto bsdf = [&](int type) {
        const float* c = type == 2 ? sh.boundary : sh.fluid;
        return v3<float>(c[0], c[1], c[2]);
    };
    int type = -1;
    V3<float> p, n;
    auto trace = [&](V3<float> o, V3<float> d, float off, bool with_sky, V3<float> sd, float sky_off, bool& occluded) {
        int ty = -1;
        V3<float> q, m;
        float len;
        if (with_sky) occluded = trace_ray<R>(o, sd, sky_off, s, cell_start, rs, sh_ray, false, ty, q, m, len);
        const bool hit = trace_ray<R>(o, d, off, s, cell_start, rs, sh_ray, true, ty, q, m, len);
        if (hit) {
            type = ty;
            p = q;
            n = m;
        }
        return hit;
    };
    V3<float> sum = v3<float>(0.f, 0.f, 0.f);
    for (int smp = 0; smp < sh.samples; smp++) {
        bool occluded;
        V3<float> out = v3<float>(0.f, 0.f, 0.f);
        if (!trace(origin, dir, rng.next() * rs.step, false, dir, 0.f, occluded)) {
            out = sh.normals_only ? v3<float>(-dir.x / 2.0f + 0.5f, -dir.y / 2.0f + 0.5f, -dir.z / 2.0f + 0.5f)
                                  : v3<float>(1.f, 1.f, 1.f);   // the sky
        } else if (sh.normals_only) {
            out = v3<float>(n.x / 2.0f + 0.5f, n.y / 2.0f + 0.5f, n.z / 2.0f + 0.5f);
        } else {
            V3<float> wgt = v3<float>(1.f, 1.f, 1.f);
            for (int depth = 0; depth < sh.max_depth; depth++) {
                if (fabsf(wgt.x) <= kFltEps && fabsf(wgt.y) <= kFltEps && fabsf(wgt.z) <= kFltEps) break;
                const V3<float> f = bsdf(type), from = n;
                // a cosine-weighted direction towards the sky, unless occluded, and the bounce
                V3<float> sd, nd;
                float sa, na;
                const float z1 = rng.next(), z2 = rng.next(), sky_off = rng.next() * rs.step;
                cosine_sample(z1, z2, n, sd, sa);
                const float z3 = rng.next(), z4 = rng.next(), off = rng.next() * rs.step;
                cosine_sample(z3, z4, n, nd, na);
                const bool hit = trace(p, nd, off, true, sd, sky_off, occluded);
                if (!occluded) {
                    const float c = sa * fminf(fmaxf(dot(from, sd), 0.0f), 1.0f);
                    out = v3<float>(out.x + c * f.x * wgt.x, out.y + c * f.y * wgt.y, out.z + c * f.z * wgt.z);
                }
                if (!hit) break;
                const float c = na * fminf(fmaxf(dot(from, nd), 0.0f), 1.0f);
                wgt = v3<float>(wgt.x * c * f.x, wgt.y * c * f.y, wgt.z * c * f.z);
            }
        }
        sum = v3<float>(sum.x + out.x, sum.y + out.y, sum.z + out.z);
    }
    if ((threadIdx.x & 31) != 0) return;
    const float inv = 1.0f / (float)sh.samples;
    radiance[3 * px] = sum.x * inv;
    radiance[3 * px + 1] = sum.y * inv;
    radiance[3 * px + 2] = sum.z * inv;
}

}  // namespace fsb
