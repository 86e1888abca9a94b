// tmpm_adjoint.cu -- differentiable rollout of the MLS-MPM substep: forward on
// the device with checkpoints, and a hand-written reverse-mode adjoint of
// G2P, the grid update and P2G (include/tmpm.h, "differentiable rollout").
//
// The forward is the reference substep (world.rs:361-467) for the corotated
// elastic material (material.rs:440-455) in a bounded domain with the
// reference's separating or sticky walls (world.rs:561-575, 632-644), on a
// dense node array covering the domain (the differentiable scenes are small
// and bounded, so no hashing is needed).  The state (x, v, C, F) is stored
// every `checkpoint_every` substeps; the backward pass replays each segment
// from its checkpoint and runs, per substep from last to first,
//   recompute P2G + grid of the substep (node mass, momentum, velocity),
//   G2P adjoint   -> adjoint of the node velocities, partial x and F adjoints,
//   grid adjoint  -> adjoint of node mass and momentum,
//   P2G adjoint   -> adjoint of the substep's input state, and dL/dE.
// The derivative of the polar factor uses, for F = R S and a skew variation
// dR = R [w]x, the identity [w]x S + S [w]x = [(tr(S) I - S) w]x, so the
// adjoint of R is F_bar += 2 R [w]x with (tr(S) I - S) w = axial(skew(R^T R_bar)).
//
// The quadratic B-spline has sum_i grad w_i = 0 and sum_i w_i dpos_i = 0, so
// the adjoint sums sum_i grad w_i s_i and sum_i w_i u_i dpos_i^T see only the
// variation of s and u over the stencil.  A loss gradient that is almost the
// same on every node would make them small differences of large f32 terms;
// they are evaluated as sum_i grad w_i (s_i - s_c) and sum_i w_i (u_i - u_c)
// dpos_i^T with s_c, u_c the values at the stencil's centre node, which is the
// same sum in exact arithmetic.

#include <atomic>
#include <climits>
#include <memory>

#include "tmpm_tile.cuh"
#include "tmpm_host.h"

using namespace tmpm;

namespace {

constexpr int kRows = 24;  // x 0-2, v 3-5, C 6-14, F 15-23 (matrices column-major: col * 3 + row)
constexpr uint32_t kErrGrid = 1u;  // a stencil left the node array


struct AdjParams {
    float h, inv_h, inv_d, dt;
    float gx, gy, gz;
    int wall_mode;
    float bmin[3], bmax[3];
    int wall_lo[3], wall_hi[3];  // wall nodes by index, as SceneParams (f64 thresholds)
    int lo[3], dim[3];  // node array: cells lo .. lo + dim - 1 per axis
    int n;
    size_t stride;      // row stride of state arrays
};

struct Consts {
    const float *mass, *vol, *radius, *damping, *nu;
    const uint8_t *fixed;
};

__device__ __forceinline__ M3f load_m(const float *S, size_t st, int row0, int i) {
    M3f m;
    m.c0 = mk(S[(row0 + 0) * st + i], S[(row0 + 1) * st + i], S[(row0 + 2) * st + i]);
    m.c1 = mk(S[(row0 + 3) * st + i], S[(row0 + 4) * st + i], S[(row0 + 5) * st + i]);
    m.c2 = mk(S[(row0 + 6) * st + i], S[(row0 + 7) * st + i], S[(row0 + 8) * st + i]);
    return m;
}
__device__ __forceinline__ void store_m(float *S, size_t st, int row0, int i, const M3f &m) {
    S[(row0 + 0) * st + i] = m.c0.x;
    S[(row0 + 1) * st + i] = m.c0.y;
    S[(row0 + 2) * st + i] = m.c0.z;
    S[(row0 + 3) * st + i] = m.c1.x;
    S[(row0 + 4) * st + i] = m.c1.y;
    S[(row0 + 5) * st + i] = m.c1.z;
    S[(row0 + 6) * st + i] = m.c2.x;
    S[(row0 + 7) * st + i] = m.c2.y;
    S[(row0 + 8) * st + i] = m.c2.z;
}
__device__ __forceinline__ V3f load_v(const float *S, size_t st, int row0, int i) {
    return mk(S[row0 * st + i], S[(row0 + 1) * st + i], S[(row0 + 2) * st + i]);
}
__device__ __forceinline__ void store_v(float *S, size_t st, int row0, int i, V3f v) {
    S[row0 * st + i] = v.x;
    S[(row0 + 1) * st + i] = v.y;
    S[(row0 + 2) * st + i] = v.z;
}
__device__ __forceinline__ M3f outer(V3f a, V3f b) { return M3f{a * b.x, a * b.y, a * b.z}; }
__device__ __forceinline__ float ddot(const M3f &a, const M3f &b) {
    return dot(a.c0, b.c0) + dot(a.c1, b.c1) + dot(a.c2, b.c2);
}
__device__ __forceinline__ float trace(const M3f &m) { return m.c0.x + m.c1.y + m.c2.z; }
__device__ __forceinline__ M3f skew_of(V3f w) {  // [w]x
    return M3f{mk(0.f, w.z, -w.y), mk(-w.z, 0.f, w.x), mk(w.y, -w.x, 0.f)};
}
// inverse transpose of m (cofactor matrix / det)
__device__ __forceinline__ M3f inv_transpose(const M3f &m, float d) {
    float inv = 1.0f / d;
    return M3f{cross(m.c1, m.c2) * inv, cross(m.c2, m.c0) * inv, cross(m.c0, m.c1) * inv};
}

struct Stencil {
    int b[3];
    float fx[3];
    float w[3][3], dw[3][3];  // [axis][offset]; dw = d w / d fx
};

__device__ __forceinline__ void stencil(V3f x, float inv_h, Stencil &s) {
    const float xs[3] = {x.x, x.y, x.z};
    for (int a = 0; a < 3; ++a) {
        s.b[a] = base_cell(xs[a], inv_h);
        float f = xs[a] * inv_h - static_cast<float>(s.b[a]);
        s.fx[a] = f;
        s.w[a][0] = 0.5f * (1.5f - f) * (1.5f - f);
        s.w[a][1] = 0.75f - (f - 1.0f) * (f - 1.0f);
        s.w[a][2] = 0.5f * (f - 0.5f) * (f - 0.5f);
        s.dw[a][0] = -(1.5f - f);
        s.dw[a][1] = -2.0f * (f - 1.0f);
        s.dw[a][2] = f - 0.5f;
    }
}

// Node index of base + offset, or -1 outside the node array.
__device__ __forceinline__ int node_at(const AdjParams &P, const Stencil &s, int a, int b, int c) {
    int lx = s.b[0] + a - P.lo[0], ly = s.b[1] + b - P.lo[1], lz = s.b[2] + c - P.lo[2];
    if (lx < 0 || ly < 0 || lz < 0 || lx >= P.dim[0] || ly >= P.dim[1] || lz >= P.dim[2]) return -1;
    return (lx * P.dim[1] + ly) * P.dim[2] + lz;
}

// ---- box tiles.  A CTA stages the nodes its particles reach (the box of
// their base cells, 2 cells wider) in shared memory: gathers read the tile
// instead of 27 global loads per particle, scatters accumulate in it in 32-bit
// fixed point (one power-of-two scale per quantity from the CTA's bounds, as in
// the transfer kernels) and flush one float4 atomic per touched node.  A CTA
// whose box does not fit, leaves the node array, or has one particle that
// dominates a bound (above 1/8 of the CTA's total) takes the direct path.
constexpr int kTileThreads = 256;
// Tile nodes of a CTA of T particles.  A chunk whose rows wrap from one lattice
// layer to the next spans the block's whole cross-section: the whole-rollout
// kernels' CTAs of 128 take 2880 nodes (45 KB), since a chunk on the direct path
// holds up every barrier.
template <int T>
constexpr int kAdjTile = T >= 256 ? 2048 : 2880;

struct TileBox {
    int lo[3], dim[3];
    int s1, s2;  // tile strides of x and y (z: 1), padded as the transfer kernels' (tile_strides)
    int nodes, ok;
};

template <int T>
struct TileSmem {
    float4 tile[kAdjTile<T>];
    int red[T / 32][6];
    float redf[T / 32][4];
};

// The part of the node array a substep's P2G writes, as six maxima that start
// at zero: [a] = P.dim - (first node - P.lo), [3 + a] = one past the last node
// - P.lo, each clipped to the array.
using NodeBounds = unsigned[6];

// Box of the valid particles' base cells, with the sums and maxima of two
// non-negative bounds over the CTA; one barrier (every warp combines the
// per-warp partials itself).
template <int T>
__device__ void tile_box(const AdjParams &P, bool valid, const int b[3], float &sa, float &sb, float &ma, float &mb,
                         TileSmem<T> &sh, TileBox &box, unsigned *bounds = nullptr) {
    int (*const red)[6] = sh.red;
    float (*const redf)[4] = sh.redf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int r[6];
    for (int a = 0; a < 3; ++a) {
        r[a] = __reduce_min_sync(0xffffffffu, valid ? b[a] : INT_MAX);
        r[3 + a] = __reduce_max_sync(0xffffffffu, valid ? b[a] : INT_MIN);
    }
    float fa = sa, fb = sb;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        fa += __shfl_xor_sync(0xffffffffu, fa, off);
        fb += __shfl_xor_sync(0xffffffffu, fb, off);
    }
    const unsigned xa = __reduce_max_sync(0xffffffffu, __float_as_uint(ma));
    const unsigned xb = __reduce_max_sync(0xffffffffu, __float_as_uint(mb));
    if (lane == 0) {
        for (int a = 0; a < 6; ++a) red[warp][a] = r[a];
        redf[warp][0] = fa;
        redf[warp][1] = fb;
        redf[warp][2] = __uint_as_float(xa);
        redf[warp][3] = __uint_as_float(xb);
    }
    __syncthreads();
    const bool mine = lane < T / 32;
    int m[6];
    for (int a = 0; a < 3; ++a) {
        m[a] = __reduce_min_sync(0xffffffffu, mine ? red[lane][a] : INT_MAX);
        m[3 + a] = __reduce_max_sync(0xffffffffu, mine ? red[lane][3 + a] : INT_MIN);
    }
    fa = mine ? redf[lane][0] : 0.0f;
    fb = mine ? redf[lane][1] : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        fa += __shfl_xor_sync(0xffffffffu, fa, off);
        fb += __shfl_xor_sync(0xffffffffu, fb, off);
    }
    sa = fa;
    sb = fb;
    ma = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(redf[lane][2]) : 0u));
    mb = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(redf[lane][3]) : 0u));
    bool ok = m[0] <= m[3];
    if (bounds && ok && threadIdx.x == 0)
        for (int a = 0; a < 3; ++a) {
            const int lo = max(m[a] - P.lo[a], 0), hi = min(m[3 + a] + 3 - P.lo[a], P.dim[a]);
            atomicMax(bounds + a, static_cast<unsigned>(max(P.dim[a] - lo, 0)));
            atomicMax(bounds + 3 + a, static_cast<unsigned>(max(hi, 0)));
        }
    int nodes = 0;
    for (int a = 0; a < 3 && ok; ++a) {
        box.lo[a] = m[a];
        box.dim[a] = m[3 + a] - m[a] + 3;
        ok = box.dim[a] <= 64 && box.lo[a] >= P.lo[a] && box.lo[a] + box.dim[a] <= P.lo[a] + P.dim[a];
    }
    if (ok) {
        tile_strides(box.dim[1], box.dim[2], box.s1, box.s2);
        nodes = box.dim[0] * box.s1;
    }
    box.nodes = nodes;
    box.ok = ok && nodes <= kAdjTile<T>;
}

// fn(t, node, count): the tile's entries four at a time, entries t .. t + count - 1
// being the nodes from `node` on (z-consecutive).
template <int T, typename Fn>
__device__ __forceinline__ void over_tile(const AdjParams &P, const TileBox &box, Fn fn) {
    const SplitP<true> split(box.s1, box.s2);
    for (int t = 4 * threadIdx.x; t < box.nodes; t += 4 * T) {
        int tx, ty, tz;
        split(t, tx, ty, tz);
        if (ty >= box.dim[1] || tz >= box.dim[2]) continue;  // padding
        fn(t, ((box.lo[0] + tx - P.lo[0]) * P.dim[1] + (box.lo[1] + ty - P.lo[1])) * P.dim[2] + (box.lo[2] + tz - P.lo[2]),
           min(4, box.dim[2] - tz));
    }
}

// The box's nodes of the dense array `src` into the tile (16-byte cp.async copies), then a barrier.
template <int T>
__device__ void fill_tile(const AdjParams &P, const TileBox &box, const float4 *src, float4 *tile) {
    over_tile<T>(P, box, [&](int t, int node, int count) {
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(tile + t));
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (e < count)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + node + e) : "memory");
    });
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

// `comps` component arrays of the scatter tile to zero.
template <int T>
__device__ __forceinline__ void zero_tile(const TileBox &box, int (*sc)[kAdjTile<T>], int comps) {
    for (int t = 4 * threadIdx.x; t < box.nodes; t += 4 * T)
        for (int c = 0; c < comps; ++c) *reinterpret_cast<int4 *>(&sc[c][t]) = make_int4(0, 0, 0, 0);
}

// Where a particle's 27 nodes are read: the CTA's tile (t0 = the particle's
// base node in it) or, without one, the dense array.
struct TileRef {
    const float4 *tile;
    int t0, s1, s2;
};
__device__ __forceinline__ TileRef tile_ref(const TileBox &box, const Stencil &s, const float4 *tile) {
    TileRef r;
    r.tile = box.ok ? tile : nullptr;
    r.s1 = box.s1;
    r.s2 = box.s2;
    r.t0 = (s.b[0] - box.lo[0]) * box.s1 + (s.b[1] - box.lo[1]) * box.s2 + (s.b[2] - box.lo[2]);
    return r;
}
// TILE: read the CTA's tile (every node of a valid particle is in it);
// otherwise the dense array, where a node outside it reads as absent.
template <bool TILE>
__device__ __forceinline__ bool node_value(const AdjParams &P, const Stencil &s, const float4 *glob, const TileRef &tr,
                                           int a, int b, int c, float4 &g) {
    if (TILE) {
        g = tr.tile[tr.t0 + a * tr.s1 + b * tr.s2 + c];
        return true;
    }
    const int id = node_at(P, s, a, b, c);
    if (id < 0) return false;
    g = __ldcg(glob + id);  // other SMs wrote it, in a whole-rollout kernel during this launch
    return true;
}

// The tile's fixed-point sums (component-major, `comps` of 4) added to the
// dense array: one float4 atomic per node with a non-zero sum.
template <int T>
__device__ void flush_tile(const AdjParams &P, const TileBox &box, int (*sc)[kAdjTile<T>], int comps, float inv0,
                           float inv1, float4 *dst) {
    over_tile<T>(P, box, [&](int t, int node, int count) {
        const int4 a = *reinterpret_cast<const int4 *>(&sc[0][t]), b = *reinterpret_cast<const int4 *>(&sc[1][t]),
                   c = *reinterpret_cast<const int4 *>(&sc[2][t]);
        const int4 d = comps > 3 ? *reinterpret_cast<const int4 *>(&sc[3][t]) : make_int4(0, 0, 0, 0);
        const int v[4][4] = {{a.x, b.x, c.x, d.x}, {a.y, b.y, c.y, d.y}, {a.z, b.z, c.z, d.z}, {a.w, b.w, c.w, d.w}};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e >= count || (v[e][0] | v[e][1] | v[e][2] | v[e][3]) == 0) continue;
            const float4 val = comps > 3 ? make_float4(v[e][0] * inv0, v[e][1] * inv1, v[e][2] * inv1, v[e][3] * inv1)
                                         : make_float4(v[e][0] * inv0, v[e][1] * inv0, v[e][2] * inv0, 0.0f);
            red_add_v4(dst + node + e, val);
        }
    });
}

__device__ __forceinline__ unsigned fx_round(float v) { return static_cast<unsigned>(__float2int_rn(v)); }

__device__ __forceinline__ void lame(float E, float nu, float &lambda, float &mu) {
    lambda = E * nu / ((1.0f + nu) * (1.0f - 2.0f * nu));
    mu = E / (2.0f * (1.0f + nu));
}

// ---------------------------------------------------------------- forward

// A particle's constants.
struct PartConst {
    float mass, vol, radius, damping, nu, E;
    bool fixed;
};
__device__ __forceinline__ PartConst load_const(const Consts &K, const float *E, int i) {
    return PartConst{K.mass[i], K.vol[i], K.radius[i], K.damping[i], K.nu[i], E[i], K.fixed[i] != 0};
}
// A particle's state, rows 0-23 of a state array.
struct PartState {
    V3f x, v;
    M3f C, F;
};
__device__ __forceinline__ PartState load_state(const float *S, size_t st, int i) {
    return PartState{load_v(S, st, 0, i), load_v(S, st, 3, i), load_m(S, st, 6, i), load_m(S, st, 15, i)};
}
__device__ __forceinline__ void store_state(float *S, size_t st, int i, const PartState &p) {
    store_v(S, st, 0, i, p.x);
    store_v(S, st, 3, i, p.v);
    store_m(S, st, 6, i, p.C);
    store_m(S, st, 15, i, p.F);
}

// P2G of a CTA's particles.  R: the polar factor of F, for the P2G adjoint of
// the same substep.  `box` returns the CTA's box, which the G2P of the same
// positions reuses.
template <int T>
__device__ __forceinline__ void p2g_chunk(const AdjParams &P, bool valid, const PartState &q, const PartConst &k,
                                          float4 *grid, uint32_t *err, M3f &R, TileSmem<T> &sh, TileBox &box,
                                          unsigned *bounds) {
    const V3f x = q.x, v = q.v;
    const M3f &C = q.C, &F = q.F;
    float lambda, mu;
    lame(k.E, k.nu, lambda, mu);
    R = polar_rotation(F);
    float J = det(F);
    M3f tau = scale(mul_bt(sub(F, R), F), 2.0f * mu);
    float iso = lambda * (J - 1.0f) * J;
    tau.c0.x += iso;
    tau.c1.y += iso;
    tau.c2.z += iso;
    const float m = k.mass;
    M3f A = add(scale(tau, -P.dt * k.vol * P.inv_d), scale(C, m));
    Stencil s;
    stencil(x, P.inv_h, s);
    // node sums are bounded by the CTA's sums of m and |m v| + 1.5 h sum |A| (weights sum to one)
    float bm = 0.0f, bp = 0.0f;
    if (valid) {
        const V3f mv = v * m;
        bm = m;
        bp = fmaxf(fmaxf(fabsf(mv.x) + 1.5f * P.h * (fabsf(A.c0.x) + fabsf(A.c1.x) + fabsf(A.c2.x)),
                         fabsf(mv.y) + 1.5f * P.h * (fabsf(A.c0.y) + fabsf(A.c1.y) + fabsf(A.c2.y))),
                   fabsf(mv.z) + 1.5f * P.h * (fabsf(A.c0.z) + fabsf(A.c1.z) + fabsf(A.c2.z)));
        if (!(bp < 1e30f)) bp = 1e30f;
    }
    float sum_m = bm, sum_p = bp, max_m = bm, max_p = bp;
    tile_box<T>(P, valid, s.b, sum_m, sum_p, max_m, max_p, sh, box, bounds);
    if (!box.ok || max_m > 0.125f * sum_m || max_p > 0.125f * sum_p) {  // direct path (CTA-uniform)
        if (!valid) return;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
                for (int c = 0; c < 3; ++c) {
                    int id = node_at(P, s, a, b, c);
                    if (id < 0) {
                        atomicOr(err, kErrGrid);
                        continue;
                    }
                    float w = s.w[0][a] * s.w[1][b] * s.w[2][c];
                    V3f dpos = mk((a - s.fx[0]) * P.h, (b - s.fx[1]) * P.h, (c - s.fx[2]) * P.h);
                    V3f mom = v * m + mul(A, dpos);
                    red_add_v4(grid + id, make_float4(w * m, w * mom.x, w * mom.y, w * mom.z));
                }
        return;
    }
    int (*sc)[kAdjTile<T>] = reinterpret_cast<int (*)[kAdjTile<T>]>(sh.tile);
    zero_tile<T>(box, sc, 4);
    __syncthreads();
    const float sm = pow2_scale(sum_m), sp = pow2_scale(sum_p);
    if (valid) {
        const int t0 = tile_ref(box, s, sh.tile).t0;
        const V3f mv = v * m;
        const float ms = m * sm;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const V3f ua = mv + A.c0 * ((a - s.fx[0]) * P.h);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const V3f uab = ua + A.c1 * ((b - s.fx[1]) * P.h);
                const float wab = s.w[0][a] * s.w[1][b];
                const int row = t0 + a * box.s1 + b * box.s2;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float w = wab * s.w[2][c], wp = w * sp;
                    const V3f u = uab + A.c2 * ((c - s.fx[2]) * P.h);
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[0][row + c]), fx_round(w * ms));
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[1][row + c]), fx_round(u.x * wp));
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[2][row + c]), fx_round(u.y * wp));
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[3][row + c]), fx_round(u.z * wp));
                }
            }
        }
    }
    __syncthreads();
    flush_tile<T>(P, box, sc, 4, pow2_inverse(sm), pow2_inverse(sp), grid);
}

// Rout (optional): the polar factors, 9 rows.
__global__ void __launch_bounds__(kTileThreads) k_p2g(AdjParams P, Consts K, const float *__restrict__ S,
                                                      const float *__restrict__ E, float4 *grid, uint32_t *err,
                                                      float *__restrict__ Rout) {
    __shared__ TileSmem<kTileThreads> sh;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    M3f R;
    TileBox box;
    p2g_chunk<kTileThreads>(P, valid, load_state(S, P.stride, ic), load_const(K, E, ic), grid, err, R, sh, box, nullptr);
    if (Rout && valid) store_m(Rout, P.stride, 0, i, R);
}

// Node velocity with the wall rule; w = bitmask of the components the walls zeroed.
__device__ __forceinline__ float4 node_velocity(const AdjParams &P, int lx, int ly, int lz, float4 mp) {
    if (!(mp.x > 0.0f)) return make_float4(0.f, 0.f, 0.f, 0.f);
    const int id[3] = {lx + P.lo[0], ly + P.lo[1], lz + P.lo[2]};
    float v[3] = {mp.y / mp.x + P.gx * P.dt, mp.z / mp.x + P.gy * P.dt, mp.w / mp.x + P.gz * P.dt};
    int mask = 0;
    for (int a = 0; a < 3; ++a) {
        const bool lower = id[a] <= P.wall_lo[a], upper = id[a] >= P.wall_hi[a];
        if (P.wall_mode == 1) {
            if (lower || upper) mask = 7;
        } else if ((lower && v[a] < 0.0f) || (upper && v[a] > 0.0f)) {
            mask |= 1 << a;
        }
    }
    for (int a = 0; a < 3; ++a)
        if (mask & (1 << a)) v[a] = 0.0f;
    return make_float4(v[0], v[1], v[2], static_cast<float>(mask));
}

__global__ void k_grid(AdjParams P, const float4 *__restrict__ grid, float4 *gv, int nodes) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    gv[i] = node_velocity(P, i / (P.dim[2] * P.dim[1]), (i / P.dim[2]) % P.dim[1], i % P.dim[2], grid[i]);
}

// Gather of one particle from the dense array: velocity, affine matrix
// (4/h^2 sum w v dpos^T).
__device__ __forceinline__ void gather_nodes(const AdjParams &P, const Stencil &s, const float4 *gv, V3f &vel, M3f &aff) {
    const TileRef none{nullptr, 0, 0, 0};
    vel = mk(0, 0, 0);
    aff = m3_zero();
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b)
            for (int c = 0; c < 3; ++c) {
                float4 g;
                if (!node_value<false>(P, s, gv, none, a, b, c, g)) continue;
                float w = s.w[0][a] * s.w[1][b] * s.w[2][c];
                V3f nv = mk(g.x, g.y, g.z);
                V3f dpos = mk((a - s.fx[0]) * P.h, (b - s.fx[1]) * P.h, (c - s.fx[2]) * P.h);
                vel = vel + nv * w;
                aff = add(aff, scale(outer(nv, dpos), w * P.inv_d));
            }
}
__device__ __forceinline__ void gather(const AdjParams &P, const Stencil &s, const float4 *gv, const TileRef &tr,
                                       V3f &vel, M3f &aff) {
    if (!tr.tile) {
        gather_nodes(P, s, gv, vel, aff);
        return;
    }
    V3f m0, m1, m2;
    gather_moments(s.w[0], s.w[1], s.w[2], [&](int a, int b) { return tr.tile + (tr.t0 + a * tr.s1 + b * tr.s2); }, vel, m0,
                   m1, m2);
    const float hd = P.h * P.inv_d;
    aff.c0 = (m0 + vel * (1.0f - s.fx[0])) * hd;
    aff.c1 = (m1 + vel * (1.0f - s.fx[1])) * hd;
    aff.c2 = (m2 + vel * (1.0f - s.fx[2])) * hd;
}

// G2P of a CTA's particles, whose box `box` holds (tile barrier inside): the
// state becomes the next substep's.
template <int T>
__device__ __forceinline__ void g2p_chunk(const AdjParams &P, bool valid, PartState &q, const PartConst &k,
                                          const float4 *gv, TileSmem<T> &sh, const TileBox &box) {
    if (box.ok) fill_tile<T>(P, box, gv, sh.tile);
    if (!valid) return;
    if (k.fixed) {
        q.v = mk(0, 0, 0);
        q.C = m3_zero();
        return;
    }
    Stencil s;
    stencil(q.x, P.inv_h, s);
    V3f vel;
    M3f aff;
    gather(P, s, gv, tile_ref(box, s, sh.tile), vel, aff);
    vel = vel * expf(-k.damping * P.dt);
    V3f pos = q.x + vel * P.dt;
    for (int a = 0; a < 3; ++a) {
        float lower = P.bmin[a] + k.radius, upper = P.bmax[a] - k.radius;
        float pa = comp(pos, a), va = comp(vel, a);
        if (pa < lower) {
            set_comp(pos, a, lower);
            set_comp(vel, a, fmaxf(va, 0.0f));
        } else if (pa > upper) {
            set_comp(pos, a, upper);
            set_comp(vel, a, fminf(va, 0.0f));
        }
    }
    q.F = mul(add(m3_identity(), scale(aff, P.dt)), q.F);
    q.x = pos;
    q.v = vel;
    q.C = aff;
}

__global__ void __launch_bounds__(kTileThreads) k_g2p(AdjParams P, Consts K, const float *__restrict__ S,
                                                      const float *__restrict__ E, float *__restrict__ Sn,
                                                      const float4 *__restrict__ gv) {
    __shared__ TileSmem<kTileThreads> sh;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    PartState q = load_state(S, P.stride, ic);
    Stencil s;
    stencil(q.x, P.inv_h, s);
    float z0 = 0.f, z1 = 0.f, z2 = 0.f, z3 = 0.f;
    TileBox box;
    tile_box<kTileThreads>(P, valid, s.b, z0, z1, z2, z3, sh, box);
    g2p_chunk<kTileThreads>(P, valid, q, load_const(K, E, ic), gv, sh, box);
    if (valid) store_state(Sn, P.stride, i, q);
}

// ---------------------------------------------------------------- adjoint

// Node sums of the two particle adjoints, over the differences d_i of a node
// vector f_i (P: momentum adjoints y, z, w; otherwise node velocities x, y, z) and
// its value at the stencil's centre f_c:
//   sum   = sum_i w_i d_i,
//   grad  = sum_i grad w_i (d_i . (u0 + U dpos_i) + m (s_i - s_c)), s the node
//           scalar x (P only),
//   m0..2 = sum_i w_i (offset - 1) d_i along x, y, z (P only),
// factored by axis as gather_moments.
template <bool TILE, bool P2G>
__device__ __forceinline__ void adjoint_sums(const AdjParams &P, const Stencil &s, const float4 *nodes, const TileRef &tr,
                                             V3f u0, const M3f &U, float m, V3f &center, V3f &sum, V3f &grad, V3f &m0,
                                             V3f &m1, V3f &m2) {
    auto vec = [](const float4 &g) { return P2G ? mk(g.y, g.z, g.w) : mk(g.x, g.y, g.z); };
    float4 gc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!node_value<TILE>(P, s, nodes, tr, 1, 1, 1, gc)) gc = make_float4(0.f, 0.f, 0.f, 0.f);
    center = vec(gc);
    sum = grad = m0 = m1 = m2 = mk(0, 0, 0);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const V3f ua = u0 + U.c0 * ((a - s.fx[0]) * P.h);
        V3f s0 = mk(0, 0, 0), s1 = s0, s2 = s0;
        float y = 0.f, yd = 0.f, yz = 0.f;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const V3f uab = ua + U.c1 * ((b - s.fx[1]) * P.h);
            V3f r = mk(0, 0, 0), rm = r;
            float q = 0.f, qd = 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float4 g;
                if (!node_value<TILE>(P, s, nodes, tr, a, b, c, g)) continue;
                const V3f d = vec(g) - center;
                const V3f u = uab + U.c2 * ((c - s.fx[2]) * P.h);
                float qi = dot(d, u);
                if (P2G) qi += m * (g.x - gc.x);
                q += s.w[2][c] * qi;
                qd += s.dw[2][c] * qi;
                const V3f wd = d * s.w[2][c];
                r = r + wd;
                if (P2G && c == 0) rm = rm - wd;
                if (P2G && c == 2) rm = rm + wd;
            }
            s0 = s0 + r * s.w[1][b];
            if (P2G) {
                if (b == 0) s1 = s1 - r * s.w[1][0];
                if (b == 2) s1 = s1 + r * s.w[1][2];
                s2 = s2 + rm * s.w[1][b];
            }
            y += s.w[1][b] * q;
            yd += s.dw[1][b] * q;
            yz += s.w[1][b] * qd;
        }
        sum = sum + s0 * s.w[0][a];
        if (P2G) {
            if (a == 0) m0 = m0 - s0 * s.w[0][0];
            if (a == 2) m0 = m0 + s0 * s.w[0][2];
            m1 = m1 + s1 * s.w[0][a];
            m2 = m2 + s2 * s.w[0][a];
        }
        grad = grad + mk(s.dw[0][a] * y, s.w[0][a] * yd, s.w[0][a] * yz);
    }
    grad = grad * P.inv_h;
}

// G2P adjoint of a CTA's particles at positions x with deformation F: `ab` is the
// adjoint of the substep's output state; xq, Fq return the partial adjoints of
// x and F, and the node-velocity adjoint is added to gvb.  `box` returns the
// CTA's box.
template <int T>
__device__ __forceinline__ void g2p_back_chunk(const AdjParams &P, bool valid, V3f x, const M3f &F,
                                               const PartConst &k, const float4 *gv, const PartState &ab, V3f &xq,
                                               M3f &Fq, float4 *gvb, TileSmem<T> &sh, TileBox &box) {
    const bool active = valid && !k.fixed;
    Stencil s;
    stencil(x, P.inv_h, s);
    float z0 = 0.f, z1 = 0.f, z2 = 0.f, z3 = 0.f;
    tile_box<T>(P, valid, s.b, z0, z1, z2, z3, sh, box);
    if (box.ok) fill_tile<T>(P, box, gv, sh.tile);
    else __syncthreads();  // every warp has read the partials before the second reduction writes them
    const TileRef tr = tile_ref(box, s, sh.tile);
    V3f velb = mk(0, 0, 0);
    M3f Cb = m3_zero();
    float bg = 0.0f;  // bound of the particle's velocity-adjoint contributions
    if (valid) {
        const V3f xb_o = ab.x, vb_o = ab.v;
        const M3f &Cb_o = ab.C, &Fb_o = ab.F;
        if (!active) {  // x and F pass through; v and C are reset
            xq = xb_o;
            Fq = Fb_o;
        } else {
            V3f vel;
            M3f aff;
            gather(P, s, gv, tr, vel, aff);
            const float ed = expf(-k.damping * P.dt);
            V3f veld = vel * ed;
            V3f pos = x + veld * P.dt;
            const float r = k.radius;
            V3f xb = xb_o;
            velb = vb_o;
            for (int a = 0; a < 3; ++a) {
                float lower = P.bmin[a] + r, upper = P.bmax[a] - r;
                float pa = comp(pos, a), va = comp(veld, a);
                if (pa < lower) {
                    set_comp(xb, a, 0.0f);
                    if (!(va > 0.0f)) set_comp(velb, a, 0.0f);
                } else if (pa > upper) {
                    set_comp(xb, a, 0.0f);
                    if (!(va < 0.0f)) set_comp(velb, a, 0.0f);
                }
            }
            velb = (velb + xb * P.dt) * ed;                       // pos = x + dt v_damped
            Cb = add(Cb_o, scale(mul_bt(Fb_o, F), P.dt));         // Fn = (I + dt C) F
            M3f Fb = mul(transpose(add(m3_identity(), scale(aff, P.dt))), Fb_o);
            // grad w (v_i . velb + 4/h^2 v_i . C_b dpos_i) - 4/h^2 w C_b^T v_i with v_i -> v_i - v_c (file header)
            V3f vc, sum, grad, m0, m1, m2;
            const M3f U = scale(Cb, P.inv_d);
            if (tr.tile) adjoint_sums<true, false>(P, s, gv, tr, velb, U, 0.0f, vc, sum, grad, m0, m1, m2);
            else adjoint_sums<false, false>(P, s, gv, tr, velb, U, 0.0f, vc, sum, grad, m0, m1, m2);
            V3f xbar = xb + grad - mul(transpose(U), sum);
            xq = xbar;
            Fq = Fb;
            // |gb_k| <= w (|velb_k| + 4/h^2 * 1.5 h sum_j |Cb_kj|), and the weights sum to one
            const float q = P.inv_d * 1.5f * P.h;
            bg = fmaxf(fmaxf(fabsf(velb.x) + q * (fabsf(Cb.c0.x) + fabsf(Cb.c1.x) + fabsf(Cb.c2.x)),
                             fabsf(velb.y) + q * (fabsf(Cb.c0.y) + fabsf(Cb.c1.y) + fabsf(Cb.c2.y))),
                       fabsf(velb.z) + q * (fabsf(Cb.c0.z) + fabsf(Cb.c1.z) + fabsf(Cb.c2.z)));
            if (!(bg < 1e30f)) bg = 1e30f;
        }
    }
    // the velocity-adjoint scatter; the reduction's barrier also ends every read of the gv tile
    float sum_g = bg, sum_0 = 0.0f, max_g = bg, max_0 = 0.0f;
    TileBox box2;
    tile_box<T>(P, active, s.b, sum_g, sum_0, max_g, max_0, sh, box2);
    const bool tiled = box.ok && !(max_g > 0.125f * sum_g);
    if (!tiled) {
        if (!active) return;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
                for (int c = 0; c < 3; ++c) {
                    int id = node_at(P, s, a, b, c);
                    if (id < 0) continue;
                    float w = s.w[0][a] * s.w[1][b] * s.w[2][c];
                    V3f dpos = mk((a - s.fx[0]) * P.h, (b - s.fx[1]) * P.h, (c - s.fx[2]) * P.h);
                    V3f gb = velb * w + mul(Cb, dpos) * (P.inv_d * w);
                    red_add_v4(gvb + id, make_float4(gb.x, gb.y, gb.z, 0.0f));
                }
        return;
    }
    int (*sc)[kAdjTile<T>] = reinterpret_cast<int (*)[kAdjTile<T>]>(sh.tile);
    zero_tile<T>(box, sc, 3);
    __syncthreads();
    const float sg = pow2_scale(sum_g);
    if (active) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const V3f ua = velb + Cb.c0 * ((a - s.fx[0]) * P.h * P.inv_d);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const V3f uab = ua + Cb.c1 * ((b - s.fx[1]) * P.h * P.inv_d);
                const float wab = s.w[0][a] * s.w[1][b] * sg;
                const int row = tr.t0 + a * box.s1 + b * box.s2;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const V3f gb = (uab + Cb.c2 * ((c - s.fx[2]) * P.h * P.inv_d)) * (wab * s.w[2][c]);
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[0][row + c]), fx_round(gb.x));
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[1][row + c]), fx_round(gb.y));
                    atomicAdd(reinterpret_cast<unsigned *>(&sc[2][row + c]), fx_round(gb.z));
                }
            }
        }
    }
    __syncthreads();
    flush_tile<T>(P, box, sc, 3, pow2_inverse(sg), pow2_inverse(sg), gvb);
}

__global__ void __launch_bounds__(kTileThreads) k_g2p_back(AdjParams P, Consts K, const float *__restrict__ S,
                                                           const float *__restrict__ E, const float4 *__restrict__ gv,
                                                           const float *__restrict__ Ab, float *__restrict__ Q,
                                                           float4 *gvb) {
    __shared__ TileSmem<kTileThreads> sh;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    const size_t st = P.stride;
    V3f xq = mk(0, 0, 0);
    M3f Fq = m3_zero();
    TileBox box;
    g2p_back_chunk<kTileThreads>(P, valid, load_v(S, st, 0, ic), load_m(S, st, 15, ic), load_const(K, E, ic), gv,
                                 load_state(Ab, st, ic), xq, Fq, gvb, sh, box);
    if (valid) {
        store_v(Q, st, 0, i, xq);
        store_m(Q, st, 15, i, Fq);
    }
}

// (m_bar, p_bar) of a node from its velocity adjoint b; gv.w: the wall mask.
__device__ __forceinline__ float4 node_back(float4 mp, float4 gv, float4 b) {
    if (!(mp.x > 0.0f)) return make_float4(0.f, 0.f, 0.f, 0.f);
    const int mask = static_cast<int>(gv.w);
    if (mask & 1) b.x = 0.0f;
    if (mask & 2) b.y = 0.0f;
    if (mask & 4) b.z = 0.0f;
    const float inv_m = 1.0f / mp.x;
    const float mbar = -(b.x * mp.y + b.y * mp.z + b.z * mp.w) * inv_m * inv_m;
    return make_float4(mbar, b.x * inv_m, b.y * inv_m, b.z * inv_m);
}

// Grid adjoint: node velocity v = p / m + g dt (walls zero some components).
// In place: gvb (velocity adjoint) becomes (m_bar, p_bar).
__global__ void k_grid_back(AdjParams P, const float4 *__restrict__ grid, const float4 *__restrict__ gv, float4 *gvb,
                            int nodes) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    gvb[i] = node_back(grid[i], gv[i], gvb[i]);
}

// P2G adjoint.  In: the substep's input state S, node (m_bar, p_bar), partial
// adjoints Q from the G2P adjoint.  Out: the adjoint of the substep's input
// state (Ain) and dL/dE accumulated into Eb.
// P2G adjoint of a CTA's particles in state q (polar factor R), whose box `box`
// holds: xq, Fq are the G2P adjoint's partials, ab returns the adjoint of the
// substep's input state, dL/dE is added to Eb.
template <int T>
__device__ __forceinline__ void p2g_back_chunk(const AdjParams &P, bool valid, const PartState &q, const PartConst &k,
                                               const M3f &R, const float4 *gmb, V3f xq, const M3f &Fq, PartState &ab,
                                               float &Eb, TileSmem<T> &sh, const TileBox &box) {
    Stencil s;
    stencil(q.x, P.inv_h, s);
    if (box.ok) fill_tile<T>(P, box, gmb, sh.tile);
    if (!valid) return;
    const TileRef tr = tile_ref(box, s, sh.tile);
    const V3f v = q.v;
    const M3f &C = q.C, &F = q.F;
    const float m = k.mass, nu = k.nu;
    float lambda, mu;
    lame(k.E, nu, lambda, mu);
    float J = det(F);
    M3f FmR_FT = mul_bt(sub(F, R), F);
    M3f tau = scale(FmR_FT, 2.0f * mu);
    float iso = lambda * (J - 1.0f) * J;
    tau.c0.x += iso;
    tau.c1.y += iso;
    tau.c2.z += iso;
    const float sc = -P.dt * k.vol * P.inv_d;
    M3f A = add(scale(tau, sc), scale(C, m));
    // grad w (m m_b + p_b . (m v + A dpos)) - w A^T p_b with m_b, p_b -> minus their
    // centre values (file header); sum_i w_i p_b = sum + p_c
    V3f pc, sum, grad, m0, m1, m2;
    if (tr.tile) adjoint_sums<true, true>(P, s, gmb, tr, v * m, A, m, pc, sum, grad, m0, m1, m2);
    else adjoint_sums<false, true>(P, s, gmb, tr, v * m, A, m, pc, sum, grad, m0, m1, m2);
    V3f xbar = xq + grad - mul(transpose(A), sum);
    M3f Fbar = Fq;
    V3f vbar = (sum + pc) * m;
    M3f Abar = M3f{(m0 + sum * (1.0f - s.fx[0])) * P.h, (m1 + sum * (1.0f - s.fx[1])) * P.h,
                   (m2 + sum * (1.0f - s.fx[2])) * P.h};
    M3f Cbar = scale(Abar, m);
    M3f taub = scale(Abar, sc);
    float trt = trace(taub);
    float mub = 2.0f * ddot(taub, FmR_FT);
    float lamb = (J - 1.0f) * J * trt;
    // d tau / d F: 2 mu (F F^T - R F^T) + lambda (J^2 - J) I
    M3f tauT = transpose(taub);
    Fbar = add(Fbar, scale(mul(add(taub, tauT), F), 2.0f * mu));
    Fbar = sub(Fbar, scale(mul(tauT, R), 2.0f * mu));
    M3f Rb = scale(mul(taub, F), -2.0f * mu);
    M3f Sm = mul(transpose(R), F);
    M3f Ssym = scale(add(Sm, transpose(Sm)), 0.5f);
    M3f G = mul(transpose(R), Rb);
    // axial vector of skew(G) = (G - G^T) / 2
    V3f kx = mk(0.5f * (G.c1.z - G.c2.y), 0.5f * (G.c2.x - G.c0.z), 0.5f * (G.c0.y - G.c1.x));
    M3f Mx = scale(Ssym, -1.0f);
    float tS = trace(Ssym);
    Mx.c0.x += tS;
    Mx.c1.y += tS;
    Mx.c2.z += tS;
    float dM = det(Mx);
    V3f om = mul(transpose(inv_transpose(Mx, dM)), kx);  // Mx^-1 k
    Fbar = add(Fbar, scale(mul(R, skew_of(om)), 2.0f));
    Fbar = add(Fbar, scale(inv_transpose(F, J), lambda * (2.0f * J - 1.0f) * trt * J));
    ab = PartState{xbar, vbar, Cbar, Fbar};
    Eb += lamb * nu / ((1.0f + nu) * (1.0f - 2.0f * nu)) + mub / (2.0f * (1.0f + nu));
}

__global__ void __launch_bounds__(kTileThreads, 2) k_p2g_back(AdjParams P, Consts K, const float *__restrict__ S,
                                                           const float *__restrict__ E, const float4 *__restrict__ gmb,
                                                           const float *__restrict__ Q, float *__restrict__ Ain,
                                                           float *__restrict__ Eb, const float *__restrict__ Rin) {
    __shared__ TileSmem<kTileThreads> sh;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    const size_t st = P.stride;
    const PartState q = load_state(S, st, ic);
    Stencil s;
    stencil(q.x, P.inv_h, s);
    float z0 = 0.f, z1 = 0.f, z2 = 0.f, z3 = 0.f;
    TileBox box;
    tile_box<kTileThreads>(P, valid, s.b, z0, z1, z2, z3, sh, box);
    PartState ab;
    float eb = 0.0f;
    p2g_back_chunk<kTileThreads>(P, valid, q, load_const(K, E, ic), load_m(Rin, st, 0, ic), gmb, load_v(Q, st, 0, ic),
                                 load_m(Q, st, 15, ic), ab, eb, sh, box);
    if (valid) {
        store_state(Ain, st, i, ab);
        Eb[i] += eb;
    }
}

// ---------------------------------------------------------------- whole rollouts

// At the sizes a differentiable rollout is built for, each kernel of a substep
// is a partial wave of latency-bound CTAs, and launches, the node-array passes
// and reloading the particles take as long as the arithmetic.  When every
// particle's thread fits on the GPU at once, the forward and the adjoint are
// therefore one cooperative launch each: thread i keeps particle i, phases are
// separated by grid-wide barriers, and the node passes visit only the part of
// the array the substep's P2G wrote (NodeBounds), which they also clear.
// Measured before (kernel by kernel, lattice order, sums node by node) and now,
// wall clock of the call in a loop of calls, host share included: 64,000
// particles x 256 substeps forward 9.4 -> 5.2 ms, adjoint 12.0 -> 8.5 ms (stepwise,
// see whole_backward_particles); 4,096 x 64 forward 1.50 -> 0.66, adjoint 1.92 ->
// 1.20 ms.  The same kernels and row order launched one by one: forward 6.0 and 1.06
// ms, adjoint of 4,096 particles 1.57 ms.
constexpr int kRolloutThreads = 128;  // 4 CTAs an SM at 128 registers: 74,496 particles on 148 SMs

// Up to this many particles the adjoint is one launch, above it the stepwise
// sweep with the segment replay on a second stream: two CTAs an SM.  Whole against
// stepwise in ms, 96 substeps, with the host's share: 512 particles 1.75 / 2.18,
// 4,096 1.75 / 2.37, 17,576 1.99 / 2.53, 32,768 2.49 / 2.71; with three CTAs on some
// SMs the two are within 4 % (39,304 3.02 / 3.08, 46,656 3.00 / 3.14, 54,872 3.15 /
// 3.23), with four the stepwise sweep is ahead or level (64,000 3.45 / 3.38, 74,088
// 3.72 / 3.74).  The forward has no replay to overlap and stays whole up to its
// room (74,088: 2.57 / 2.75).
size_t whole_backward_particles() { return static_cast<size_t>(2 * device_sm_count()) * kRolloutThreads; }

struct RolloutArgs {
    const float *E;
    float *ckpt;
    float4 *grid, *gv;  // grid: zero outside a P2G and its grid update
    unsigned *bounds;   // NodeBounds of each substep, zero at launch
    uint32_t *err, *arrived;
    uint32_t substeps, every;
    size_t nodes;
    // forward: the initial state (24 rows) and the final one (rows 0-5 are written)
    const float *initial;
    float *final_state;
    // adjoint: the replay's buffers (two sets of a segment), the node adjoints
    // (gvb: zero outside a G2P adjoint and its grid adjoint), the loss gradient
    // of the final state, and the results
    float *seg[2], *seg_R[2];
    float4 *seg_grid[2], *seg_gv[2];
    float4 *gvb, *gmb;
    const float *adj_in;
    float *adj_out, *Ebar;
};

// fn(node, lx, ly, lz) over the nodes of `bounds`, spread over the grid's threads.
template <typename Fn>
__device__ __forceinline__ void over_bounds(const AdjParams &P, const unsigned *bounds, Fn fn) {
    int lo[3], n[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = P.dim[a] - static_cast<int>(__ldcg(bounds + a));
        n[a] = static_cast<int>(__ldcg(bounds + 3 + a)) - lo[a];
    }
    if (n[0] <= 0 || n[1] <= 0 || n[2] <= 0) return;
    const int total = n[0] * n[1] * n[2];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int q = t / n[2], lz = lo[2] + t - q * n[2];
        const int r = q / n[1], ly = lo[1] + q - r * n[1], lx = lo[0] + r;
        fn((lx * P.dim[1] + ly) * P.dim[2] + lz, lx, ly, lz);
    }
}

template <int T>
__global__ void __launch_bounds__(T, 512 / T) k_rollout_forward(AdjParams P, Consts K, RolloutArgs B) {
    __shared__ TileSmem<T> sh;
    const int i = blockIdx.x * T + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    const size_t st = P.stride;
    const PartConst k = load_const(K, B.E, ic);
    PartState q = load_state(B.initial, st, ic);
    uint32_t target = 0;
    TileBox box;
    M3f R;
    for (uint32_t s = 0; s < B.substeps; ++s) {
        if (valid && s % B.every == 0) store_state(B.ckpt + (s / B.every) * (kRows * st), st, i, q);
        unsigned *const bounds = B.bounds + 6 * s;
        p2g_chunk<T>(P, valid, q, k, B.grid, B.err, R, sh, box, bounds);
        if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
        over_bounds(P, bounds, [&](int node, int lx, int ly, int lz) {
            const float4 mp = __ldcg(B.grid + node);
            B.grid[node] = make_float4(0.f, 0.f, 0.f, 0.f);
            B.gv[node] = node_velocity(P, lx, ly, lz, mp);
        });
        if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
        g2p_chunk<T>(P, valid, q, k, B.gv, sh, box);
    }
    if (valid) {
        store_v(B.final_state, st, 0, i, q.x);
        store_v(B.final_state, st, 3, i, q.v);
    }
}

// The adjoint: while segment sg is swept backwards, segment sg - 1 is replayed
// from its checkpoint into the other buffer set; a substep of each shares a
// pair of phases (particles, nodes).  A particle's P2G adjoint of substep s + 1
// and G2P adjoint of substep s run in one phase, its adjoint state in registers.
template <int T>
__global__ void __launch_bounds__(T, 512 / T) k_rollout_backward(AdjParams P, Consts K, RolloutArgs B) {
    __shared__ TileSmem<T> sh;
    const int i = blockIdx.x * T + threadIdx.x;
    const bool valid = i < P.n;
    const int ic = valid ? i : 0;
    const size_t st = P.stride, sf = kRows * st;
    const PartConst k = load_const(K, B.E, ic);
    uint32_t target = 0;
    TileBox box_s, box_r;  // of the sweep's substep, of the replay's

    // replay substep j of segment sg into set sg & 1
    auto replay_particles = [&](int sg, uint32_t j) {
        const int set = sg & 1;
        PartState q;
        // The sweep's particles ran just before, in the same phase.  Without a
        // tile their last shared-memory access is a read of the reduction's
        // partials, which the reduction below writes; with one it is of the tile.
        __syncthreads();
        if (j == 0) {
            q = load_state(B.ckpt + sg * sf, st, ic);
        } else {
            q = load_state(B.seg[set] + (j - 1) * sf, st, ic);
            g2p_chunk<T>(P, valid, q, k, B.seg_gv[set] + (j - 1) * B.nodes, sh, box_r);
        }
        if (valid) store_state(B.seg[set] + j * sf, st, i, q);
        M3f R;
        p2g_chunk<T>(P, valid, q, k, B.grid, B.err, R, sh, box_r, B.bounds + 6 * (sg * B.every + j));
        if (valid) store_m(B.seg_R[set] + j * 9 * st, st, 0, i, R);
    };
    auto replay_nodes = [&](int sg, uint32_t j) {
        const int set = sg & 1;
        float4 *const g = B.seg_grid[set] + j * B.nodes, *const v = B.seg_gv[set] + j * B.nodes;
        over_bounds(P, B.bounds + 6 * (sg * B.every + j), [&](int node, int lx, int ly, int lz) {
            const float4 mp = __ldcg(B.grid + node);
            B.grid[node] = make_float4(0.f, 0.f, 0.f, 0.f);
            g[node] = mp;
            v[node] = node_velocity(P, lx, ly, lz, mp);
        });
    };
    // the P2G adjoint of substep s, whose node adjoints are in gmb: ab becomes
    // the adjoint of its input state
    PartState ab = load_state(B.adj_in, st, ic);
    V3f xq = mk(0, 0, 0);
    M3f Fq = m3_zero();
    float Eb = 0.0f;
    auto p2g_adjoint = [&](uint32_t s) {
        const int set = (s / B.every) & 1;
        const uint32_t j = s % B.every;
        p2g_back_chunk<T>(P, valid, load_state(B.seg[set] + j * sf, st, ic), k,
                          load_m(B.seg_R[set] + j * 9 * st, st, 0, ic), B.gmb, xq, Fq, ab, Eb, sh, box_s);
    };

    const int segments = static_cast<int>((B.substeps + B.every - 1) / B.every);
    const uint32_t tail = B.substeps - (segments - 1) * B.every;
    for (uint32_t j = 0; j < tail; ++j) {
        replay_particles(segments - 1, j);
        if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
        replay_nodes(segments - 1, j);
        if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
    }
    for (int sg = segments - 1; sg >= 0; --sg) {
        const int set = sg & 1;
        const uint32_t s0 = sg * B.every, sweep = min(B.substeps - s0, B.every), replay = sg > 0 ? B.every : 0;
        for (uint32_t t = 0; t < max(sweep, replay); ++t) {
            const uint32_t s = s0 + sweep - 1 - t, j = s - s0;
            if (t < sweep) {
                if (s + 1 < B.substeps) p2g_adjoint(s + 1);
                const float *S = B.seg[set] + j * sf;
                g2p_back_chunk<T>(P, valid, load_v(S, st, 0, ic), load_m(S, st, 15, ic), k, B.seg_gv[set] + j * B.nodes,
                                  ab, xq, Fq, B.gvb, sh, box_s);
            }
            if (t < replay) replay_particles(sg - 1, t);
            if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
            if (t < sweep) {
                const float4 *const g = B.seg_grid[set] + j * B.nodes, *const v = B.seg_gv[set] + j * B.nodes;
                over_bounds(P, B.bounds + 6 * s, [&](int node, int, int, int) {
                    const float4 b = __ldcg(B.gvb + node);
                    B.gvb[node] = make_float4(0.f, 0.f, 0.f, 0.f);
                    B.gmb[node] = node_back(__ldcg(g + node), __ldcg(v + node), b);
                });
            }
            if (t < replay) replay_nodes(sg - 1, t);
            if (!grid_barrier(B.arrived, target += gridDim.x, B.err)) return;
        }
    }
    p2g_adjoint(0);
    if (valid) {
        store_v(B.adj_out, st, 3, i, ab.v);
        B.Ebar[i] = Eb;
    }
}
}  // namespace

struct TmpmAdjoint {
    int device = 0;
    cudaStream_t stream = nullptr;
    TmpmParams params{};
    double dt = 0.0;
    uint32_t substeps = 0, every = 16;
    HostWorld world;     // initial state (velocity and E replaced per forward)
    size_t n = 0;
    AdjParams P{};
    int nodes = 0;
    std::vector<uint32_t> order;  // device row -> particle (rollout_order)
    DevBuf<float> mass, vol, radius, damping, nu, E, Ebar;
    DevBuf<uint8_t> fixed;
    DevBuf<float> ckpt, adj[2], part;
    DevBuf<float> initial;  // the initial state; its velocity rows are written per forward
    PinnedBuf staging;      // rows copied to and from the device
    DevBuf<float4> grid, gv, gvb, gmb;
    DevBuf<unsigned> bounds;  // whole-rollout kernels: NodeBounds per substep, and the barrier word
    // one cooperative launch each (k_rollout_forward, k_rollout_backward), until one is refused (replay)
    bool whole_forward = false, whole_backward = false;
    // Two buffer sets for replayed segments (segment sg uses set sg & 1): per
    // substep of the segment, its state, the grid after P2G (mass and
    // momentum), the node velocities and the particles' polar factors, so the
    // adjoint sweep reuses them instead of recomputing P2G and the grid
    // update.  The forward ping-pongs between the first two states of set 0.
    DevBuf<float> seg[2];
    DevBuf<float4> seg_grid[2], seg_gv[2];
    DevBuf<float> seg_R[2];
    DevBuf<uint32_t> err;
    bool have_forward = false;
    std::string last_error;
    // The forward and adjoint sweeps (fixed launches over fixed buffers) are
    // captured as CUDA graphs on first use and replayed afterwards.
    cudaGraphExec_t fwd_exec = nullptr, bwd_exec = nullptr;
    // The adjoint sweep replays segment sg - 1 on `side` while `stream` runs the
    // adjoint of segment sg: at the sizes this rollout is built for, each
    // kernel fills less than one wave of the GPU, so the two overlap.
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_replayed = nullptr, ev_swept = nullptr;

    ~TmpmAdjoint() {
        if (stream) cudaStreamSynchronize(stream);
        if (side) cudaStreamSynchronize(side);
        if (fwd_exec) cudaGraphExecDestroy(fwd_exec);
        if (bwd_exec) cudaGraphExecDestroy(bwd_exec);
        for (cudaEvent_t ev : {ev_fork, ev_replayed, ev_swept})
            if (ev) cudaEventDestroy(ev);
        if (side) cudaStreamDestroy(side);
        if (stream) cudaStreamDestroy(stream);
    }

    // Capture `launch` (stream work only) into *exec; a launch that was refused
    // is an error although the capture may have gone on without it.
    template <typename Fn>
    cudaError_t capture(cudaGraphExec_t *exec, Fn launch) {
        cudaGraph_t g = nullptr;
        cudaGetLastError();  // an error of an earlier call is not this capture's
        cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
        if (e) return e;
        launch();
        const cudaError_t launched = cudaGetLastError();
        e = cudaStreamEndCapture(stream, &g);
        if (launched) e = launched;
        if (!e) e = cudaGraphInstantiate(exec, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e) *exec = nullptr;
        return e;
    }

    // Launch a sweep's graph, captured on first use.  `whole`: as one cooperative
    // launch.  The device may refuse that where the occupancy query did not say so
    // (fewer SMs open to the process than the device has): the sweep then runs
    // kernel by kernel, now and in later calls.
    template <typename Whole, typename Stepwise>
    cudaError_t replay(cudaGraphExec_t *exec, bool &whole, Whole launch_once, Stepwise launch_steps) {
        cudaError_t e;
        if (whole) {
            e = *exec ? cudaSuccess : capture(exec, launch_once);
            if (!e) e = cudaGraphLaunch(*exec, stream);
            if (!e) return e;
            cudaGetLastError();
            if (*exec) cudaGraphExecDestroy(*exec);
            *exec = nullptr;
            whole = false;
        }
        if (!*exec && (e = capture(exec, launch_steps))) return e;
        return cudaGraphLaunch(*exec, stream);
    }

    // Arguments of the whole-rollout kernels, whose work arrays start at zero.
    RolloutArgs rollout_args() {
        RolloutArgs B{};
        B.E = E.ptr;
        B.ckpt = ckpt.ptr;
        B.grid = grid.ptr;
        B.gv = gv.ptr;
        B.bounds = bounds.ptr;
        B.arrived = bounds.ptr + 6 * static_cast<size_t>(substeps);
        B.err = err.ptr;
        B.substeps = substeps;
        B.every = every;
        B.nodes = nodes;
        B.initial = initial.ptr;
        B.final_state = seg[0].ptr + (substeps % 2) * state_floats();
        for (int set = 0; set < 2; ++set) {
            B.seg[set] = seg[set].ptr;
            B.seg_R[set] = seg_R[set].ptr;
            B.seg_grid[set] = seg_grid[set].ptr;
            B.seg_gv[set] = seg_gv[set].ptr;
        }
        B.gvb = gvb.ptr;
        B.gmb = gmb.ptr;
        B.adj_in = adj[0].ptr;
        B.adj_out = adj[substeps & 1u].ptr;
        B.Ebar = Ebar.ptr;
        return B;
    }
    template <typename Kernel>
    void launch_whole(Kernel kernel) {
        AdjParams p = P;
        Consts c = consts();
        RolloutArgs B = rollout_args();
        cudaMemsetAsync(grid.ptr, 0, sizeof(float4) * nodes, stream);
        cudaMemsetAsync(bounds.ptr, 0, sizeof(unsigned) * bounds.count, stream);
        void *args[] = {&p, &c, &B};
        cudaLaunchCooperativeKernel(kernel, dim3(static_cast<unsigned>((n + kRolloutThreads - 1) / kRolloutThreads)),
                                    dim3(kRolloutThreads), args, 0, stream);
    }
    // Particles whose threads are all resident at once in a whole-rollout kernel.
    template <typename Kernel>
    static size_t whole_room(Kernel kernel) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRolloutThreads, 0)) {
            cudaGetLastError();
            return 0;
        }
        return static_cast<size_t>(whole_launch_room(per_sm * device_sm_count())) * kRolloutThreads;
    }

    // The forward sweep, kernel by kernel: `substeps` substeps from the initial
    // state in seg[0] (its first state) ping-ponging with its second state, a
    // checkpoint every `every`.
    void forward_sweep() {
        cudaMemcpyAsync(seg[0].ptr, initial.ptr, sizeof(float) * state_floats(), cudaMemcpyDeviceToDevice, stream);
        float *cur = seg[0].ptr, *nxt = seg[0].ptr + state_floats();
        for (uint32_t s = 0; s < substeps; ++s) {
            if (s % every == 0)
                cudaMemcpyAsync(ckpt.ptr + (s / every) * state_floats(), cur, sizeof(float) * state_floats(),
                                cudaMemcpyDeviceToDevice, stream);
            substep(cur, nxt);
            std::swap(cur, nxt);
        }
    }

    // Replay segment sg from its checkpoint into buffer set sg & 1 on stream st:
    // per substep j its state, grid, node velocities and polar factors.
    void replay_segment(int sg, cudaStream_t st) {
        const int set = sg & 1;
        const uint32_t s0 = sg * every, s1 = std::min(substeps, s0 + every);
        float *S = seg[set].ptr;
        cudaMemcpyAsync(S, ckpt.ptr + sg * state_floats(), sizeof(float) * state_floats(), cudaMemcpyDeviceToDevice,
                        st);
        for (uint32_t s = s0; s < s1; ++s) {
            const uint32_t j = s - s0;
            float4 *g = seg_grid[set].ptr + static_cast<size_t>(j) * nodes;
            float4 *v = seg_gv[set].ptr + static_cast<size_t>(j) * nodes;
            p2g_grid(S + j * state_floats(), g, v, seg_R[set].ptr + static_cast<size_t>(j) * 9 * n, st);
            if (s + 1 < s1)
                k_g2p<<<blocks_n(), kTileThreads, 0, st>>>(P, consts(), S + j * state_floats(),
                                                           E.ptr, S + (j + 1) * state_floats(), v);
        }
    }

    // The adjoint of segment sg (replayed into set sg & 1), substep by substep
    // from its last; `a` is the adj buffer holding the adjoint of its final state.
    void sweep_segment(int sg, int &a) {
        const int set = sg & 1;
        const uint32_t s0 = sg * every, s1 = std::min(substeps, s0 + every);
        for (int s = static_cast<int>(s1) - 1; s >= static_cast<int>(s0); --s) {
            const uint32_t j = s - s0;
            const float *S = seg[set].ptr + j * state_floats();
            const float4 *g = seg_grid[set].ptr + static_cast<size_t>(j) * nodes;
            const float4 *v = seg_gv[set].ptr + static_cast<size_t>(j) * nodes;
            cudaMemsetAsync(gvb.ptr, 0, sizeof(float4) * nodes, stream);
            k_g2p_back<<<blocks_n(), kTileThreads, 0, stream>>>(P, consts(), S, E.ptr, v, adj[a].ptr, part.ptr, gvb.ptr);
            k_grid_back<<<blocks_nodes(), 256, 0, stream>>>(P, g, v, gvb.ptr, nodes);
            k_p2g_back<<<blocks_n(), kTileThreads, 0, stream>>>(P, consts(), S, E.ptr, gvb.ptr, part.ptr, adj[a ^ 1].ptr,
                                                                Ebar.ptr, seg_R[set].ptr + static_cast<size_t>(j) * 9 * n);
            a ^= 1;
        }
    }

    void backward_whole() {
        cudaMemsetAsync(gvb.ptr, 0, sizeof(float4) * nodes, stream);
        launch_whole(k_rollout_backward<kRolloutThreads>);
    }

    // The adjoint sweep, kernel by kernel, from adj[0] (the loss gradient of the final state),
    // segment by segment from the last checkpoint back; the initial-state
    // adjoint ends in adj[substeps & 1].  Segment sg - 1 is replayed on `side`
    // while `stream` sweeps segment sg; the replay into a set waits for the
    // sweep that last read it (segment sg + 1), and each sweep for its replay.
    void backward_sweep() {
        int a = 0;
        const int segments = static_cast<int>((substeps + every - 1) / every);
        cudaEventRecord(ev_fork, stream);
        cudaStreamWaitEvent(side, ev_fork, 0);
        replay_segment(segments - 1, side);
        cudaEventRecord(ev_replayed, side);
        for (int sg = segments - 1; sg >= 0; --sg) {
            cudaStreamWaitEvent(stream, ev_replayed, 0);
            if (sg >= 1) {
                if (sg + 1 < segments) cudaStreamWaitEvent(side, ev_swept, 0);
                replay_segment(sg - 1, side);
                cudaEventRecord(ev_replayed, side);
            }
            sweep_segment(sg, a);
            cudaEventRecord(ev_swept, stream);
        }
        // every replay on `side` ends before a sweep that `stream` waits for
    }
    TmpmStatus fail(TmpmStatus st, const std::string &msg) {
        last_error = msg;
        g_last_error = msg;
        return st;
    }
    TmpmStatus cuda_fail(cudaError_t e, const char *what) {
        return fail(TMPM_ERR_DEVICE, std::string(what) + ": " + cudaGetErrorString(e));
    }
    Consts consts() const { return Consts{mass.ptr, vol.ptr, radius.ptr, damping.ptr, nu.ptr, fixed.ptr}; }
    size_t state_floats() const { return kRows * n; }
    int blocks_n() const { return static_cast<int>((n + kTileThreads - 1) / kTileThreads); }
    int blocks_nodes() const { return (nodes + 255) / 256; }

    // P2G + grid of state S into g / v (and the polar factors into R when given).
    void p2g_grid(const float *S, float4 *g, float4 *v, float *R, cudaStream_t st) {
        cudaMemsetAsync(g, 0, sizeof(float4) * nodes, st);
        k_p2g<<<blocks_n(), kTileThreads, 0, st>>>(P, consts(), S, E.ptr, g, err.ptr, R);
        k_grid<<<blocks_nodes(), 256, 0, st>>>(P, g, v, nodes);
    }
    void substep(const float *S, float *Sn) {
        p2g_grid(S, grid.ptr, gv.ptr, nullptr, stream);
        k_g2p<<<blocks_n(), kTileThreads, 0, stream>>>(P, consts(), S, E.ptr, Sn, gv.ptr);
    }

    TmpmStatus check_err() {
        uint32_t e = 0;
        cudaError_t ce = cudaMemcpy(&e, err.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost);
        if (ce) return cuda_fail(ce, "adjoint status");
        if (e & kStatusTimeout) return fail(TMPM_ERR_READBACK, "a bounded device wait gave up");
        if (e & kErrGrid) return fail(TMPM_ERR_CAPACITY, "a particle stencil left the domain's node array");
        return TMPM_OK;
    }

    // fn(begin, end) over the particles on the host threads: a few thousand
    // particles a chunk are worth a thread here (random access to f64 rows).
    template <typename Fn>
    void each_range(Fn fn) {
        parallel_chunks(n, [&](size_t, size_t lo, size_t hi) { fn(lo, hi); }, 4096);
    }

    TmpmStatus forward(const double *v0, const double *young, double *x_out, double *v_out) {
        // inputs -> the host world (for the CFL check), and the velocity and
        // modulus rows; the rest of the initial state is on the device already
        ++world.version;
        if (!staging.ensure(6 * n * sizeof(float))) return fail(TMPM_ERR_DEVICE, "cudaMallocHost staging failed");
        float *const h = static_cast<float *>(staging.ptr);  // rows 0-2 velocity, 3 Young's modulus
        std::atomic<int> bad{0};
        each_range([&](size_t lo, size_t hi) {
            for (size_t i = lo; i < hi; ++i) {
                const double e = young ? young[i] : world.mparams[5 * i];
                if (!std::isfinite(e) || !(e > 0.0)) {
                    bad.fetch_or(1);
                    return;
                }
                world.mparams[5 * i] = e;
                if (v0)
                    for (int k = 0; k < 3; ++k) world.vel[3 * i + k] = v0[3 * i + k];
                if (!valid_particle(world, i)) bad.fetch_or(2);
            }
        });
        if (bad & 1) return fail(TMPM_ERR_MPM_INVALID_INPUT, "young's modulus must be positive");
        if (bad) return fail(TMPM_ERR_MPM_INVALID_INPUT, "invalid MPM input");
        if (dt > stable_timestep(world, params))
            return fail(TMPM_ERR_INVALID_INPUT, "substep dt is above the CFL bound for these inputs");
        each_range([&](size_t lo, size_t hi) {
            for (size_t j = lo; j < hi; ++j) {
                const size_t i = order[j];
                for (int k = 0; k < 3; ++k) h[k * n + j] = static_cast<float>(world.vel[3 * i + k]);
                h[3 * n + j] = static_cast<float>(world.mparams[5 * i]);
            }
        });
        cudaError_t e;
        if ((e = cudaMemcpyAsync(initial.ptr + 3 * n, h, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemcpyAsync(E.ptr, h + 3 * n, sizeof(float) * n, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemsetAsync(err.ptr, 0, sizeof(uint32_t), stream)))
            return cuda_fail(e, "adjoint upload");
        // seg[0] holds two ping-pong states during the forward; the final state
        // is in the first of them after an even number of substeps
        if ((e = replay(&fwd_exec, whole_forward, [&]() { launch_whole(k_rollout_forward<kRolloutThreads>); },
                        [&]() { forward_sweep(); })))
            return cuda_fail(e, "adjoint forward");
        const float *cur = (substeps % 2 == 0) ? seg[0].ptr : seg[0].ptr + state_floats();
        if ((e = cudaMemcpyAsync(h, cur, sizeof(float) * 6 * n, cudaMemcpyDeviceToHost, stream)) ||
            (e = cudaStreamSynchronize(stream)))
            return cuda_fail(e, "adjoint forward");
        TmpmStatus st = check_err();
        if (st != TMPM_OK) return st;
        each_range([&](size_t lo, size_t hi) {
            for (size_t j = lo; j < hi; ++j)
                for (int k = 0; k < 6; ++k)
                    if (!std::isfinite(h[k * n + j])) bad.fetch_or(4);
        });
        if (bad) return fail(TMPM_ERR_NON_FINITE_STATE, "MPM integration produced a non-finite state");
        each_range([&](size_t lo, size_t hi) {
            for (size_t j = lo; j < hi; ++j) {
                const size_t i = order[j];
                for (int k = 0; k < 3; ++k) {
                    if (x_out) x_out[3 * i + k] = h[k * n + j];
                    if (v_out) v_out[3 * i + k] = h[(3 + k) * n + j];
                }
            }
        });
        have_forward = true;
        return TMPM_OK;
    }

    TmpmStatus backward(const double *x_grad, const double *v_grad, double *v0_grad, double *young_grad) {
        if (!have_forward) return fail(TMPM_ERR_INVALID_INPUT, "backward needs a forward run first");
        if (!staging.ensure(6 * n * sizeof(float))) return fail(TMPM_ERR_DEVICE, "cudaMallocHost staging failed");
        float *const h = static_cast<float *>(staging.ptr);
        each_range([&](size_t lo, size_t hi) {
            for (size_t j = lo; j < hi; ++j) {
                const size_t i = order[j];
                for (int k = 0; k < 3; ++k) {
                    h[k * n + j] = x_grad ? static_cast<float>(x_grad[3 * i + k]) : 0.0f;
                    h[(3 + k) * n + j] = v_grad ? static_cast<float>(v_grad[3 * i + k]) : 0.0f;
                }
            }
        });
        cudaError_t e;
        // the loss gradient: positions and velocities; none on the affine matrix and F
        if ((e = cudaMemcpyAsync(adj[0].ptr, h, sizeof(float) * 6 * n, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemsetAsync(adj[0].ptr + 6 * n, 0, sizeof(float) * (state_floats() - 6 * n), stream)) ||
            (e = cudaMemsetAsync(Ebar.ptr, 0, sizeof(float) * n, stream)) ||
            (e = cudaMemsetAsync(err.ptr, 0, sizeof(uint32_t), stream)))
            return cuda_fail(e, "adjoint upload");
        // the parity of the final adj buffer: one flip per substep
        const int a = static_cast<int>(substeps & 1u);
        if ((e = replay(&bwd_exec, whole_backward, [&]() { backward_whole(); }, [&]() { backward_sweep(); })))
            return cuda_fail(e, "adjoint backward");
        float *const vb = h, *const eb = h + 3 * n;
        if ((e = cudaMemcpyAsync(vb, adj[a].ptr + 3 * n, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost, stream)) ||
            (e = cudaMemcpyAsync(eb, Ebar.ptr, sizeof(float) * n, cudaMemcpyDeviceToHost, stream)) ||
            (e = cudaStreamSynchronize(stream)))
            return cuda_fail(e, "adjoint backward");
        TmpmStatus st = check_err();
        if (st != TMPM_OK) return st;
        std::atomic<bool> bad{false};
        each_range([&](size_t lo, size_t hi) {
            for (size_t j = lo; j < hi; ++j) {
                const size_t i = order[j];
                for (int k = 0; k < 3; ++k) {
                    if (!std::isfinite(vb[k * n + j])) bad = true;
                    if (v0_grad) v0_grad[3 * i + k] = vb[k * n + j];
                }
                if (!std::isfinite(eb[j])) bad = true;
                if (young_grad) young_grad[i] = eb[j];
            }
        });
        if (bad) return fail(TMPM_ERR_NON_FINITE_STATE, "non-finite adjoint");
        return TMPM_OK;
    }
};

// Device row -> particle.  Bricks of 2 x 2 x 4 cells (a CTA's 128 particles at 8
// per cell), counted from the particles' own lowest cell and taken in a snake
// along z, then y, then x: consecutive bricks always share a face, so a chunk
// that begins inside one still has a compact box of nodes (Morton order jumps
// between octants, and such chunks left the tile: 17,576 particles 21.9 us a
// forward substep where 8,000 took 11.7).  Each full chunk of T rows is
// transposed as a session's rows are (lane_cell), so that a warp's particles fall
// on different nodes.  The order is taken once: the particles of a rollout stay
// near their neighbours.
static std::vector<uint32_t> rollout_order(const HostWorld &w, const AdjParams &P, int T) {
    const size_t n = w.n;
    HostVec<uint64_t> key(n), key2(n);
    HostVec<uint32_t> idx(n), idx2(n);
    auto cell = [&](size_t i, int a) {
        // inside the node array for every valid particle; clamped, since it only orders rows
        const float c = std::floor(static_cast<float>(w.pos[3 * i + a]) * P.inv_h - 0.5f);
        return std::min(std::max(static_cast<int>(c), P.lo[a]), P.lo[a] + P.dim[a] - 1);
    };
    struct Range {
        int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    };
    constexpr size_t kChunk = 4096;  // particles worth a host thread
    std::vector<Range> part(host_threads() + 1);
    parallel_chunks(n, [&](size_t c, size_t begin, size_t end) {
        Range r;
        for (size_t i = begin; i < end; ++i)
            for (int a = 0; a < 3; ++a) {
                const int v = cell(i, a);
                r.lo[a] = std::min(r.lo[a], v);
                r.hi[a] = std::max(r.hi[a], v);
            }
        part[c] = r;
    }, kChunk);
    Range all_cells;
    for (const Range &r : part)
        for (int a = 0; a < 3; ++a) {
            all_cells.lo[a] = std::min(all_cells.lo[a], r.lo[a]);
            all_cells.hi[a] = std::max(all_cells.hi[a], r.hi[a]);
        }
    const int *lo = all_cells.lo, *hi = all_cells.hi;
    const uint64_t nx = ((hi[0] - lo[0]) >> 1) + 1, ny = ((hi[1] - lo[1]) >> 1) + 1, nz = ((hi[2] - lo[2]) >> 2) + 1;
    parallel_chunks(n, [&](size_t, size_t begin, size_t end) {
        for (size_t i = begin; i < end; ++i) {
            const uint64_t x = cell(i, 0) - lo[0], y = cell(i, 1) - lo[1], z = cell(i, 2) - lo[2];
            const uint64_t by = y >> 1, bz = z >> 2, row = (x >> 1) * ny + ((x >> 1) & 1 ? ny - 1 - by : by);
            const uint64_t in = (z & 2) << 2 | (x & 1) << 2 | (y & 1) << 1 | (z & 1);
            key[i] = (row * nz + (row & 1 ? nz - 1 - bz : bz)) << 4 | in;
            idx[i] = static_cast<uint32_t>(i);
        }
    }, kChunk);
    const uint64_t all = nx * ny * nz << 4;  // above every key
    for (int shift = 0; shift < 64 && (all >> shift) != 0; shift += 11) {  // stable LSD radix passes
        std::vector<uint32_t> at(2049, 0);
        for (size_t i = 0; i < n; ++i) ++at[((key[i] >> shift) & 2047) + 1];
        for (int d = 0; d < 2048; ++d) at[d + 1] += at[d];
        for (size_t i = 0; i < n; ++i) {
            const uint32_t to = at[(key[i] >> shift) & 2047]++;
            key2[to] = key[i];
            idx2[to] = idx[i];
        }
        key.swap(key2);
        idx.swap(idx2);
    }
    std::vector<uint32_t> rows(n);
    for (size_t j = 0; j < n; ++j) {
        const size_t chunk = j / T, kk = j % T;
        const size_t sj = (chunk + 1) * T <= n ? chunk * T + lane_cell(static_cast<int>(kk % 32)) * (T / 32) + kk / 32 : j;
        rows[j] = idx[sj];
    }
    return rows;
}

extern "C" {

TmpmStatus tmpm_adjoint_create(const TmpmParams *params, const TmpmParticleArrays *particles, double substep_dt,
                               uint32_t substeps, uint32_t checkpoint_every, int32_t device, TmpmAdjoint **out) {
    if (!out || !params) {
        g_last_error = "null argument";
        return TMPM_ERR_INVALID_INPUT;
    }
    *out = nullptr;
    if (!params_valid(*params)) {
        g_last_error = "invalid MPM input";
        return TMPM_ERR_MPM_INVALID_INPUT;
    }
    if (!params->has_bounds) {
        g_last_error = "the differentiable rollout needs a bounded domain";
        return TMPM_ERR_INVALID_INPUT;
    }
    if (substeps == 0 || checkpoint_every == 0) {
        g_last_error = "substeps and checkpoint interval must be positive";
        return TMPM_ERR_INVALID_INPUT;
    }
    auto a = std::make_unique<TmpmAdjoint>();
    std::string err;
    TmpmStatus st = load_checked(particles, a->world, err);
    if (st != TMPM_OK) {
        g_last_error = err;
        return st;
    }
    HostWorld &w = a->world;
    if (w.n == 0 || w.n > (1u << 26)) {
        g_last_error = "particle count must be 1 .. 2^26";
        return TMPM_ERR_INVALID_INPUT;
    }
    for (size_t i = 0; i < w.n; ++i) {
        if (w.material[i] != TMPM_MAT_ELASTIC || !w.enabled[i]) {
            g_last_error = "the differentiable rollout takes enabled corotated elastic particles";
            return TMPM_ERR_INVALID_INPUT;
        }
        for (int k = 0; k < 3; ++k)
            if (!(w.pos[3 * i + k] >= params->bounds_min[k] && w.pos[3 * i + k] <= params->bounds_max[k])) {
                g_last_error = "particles must start inside the domain bounds";
                return TMPM_ERR_INVALID_INPUT;
            }
    }
    if (!std::isfinite(substep_dt) || substep_dt <= 0.0 || substep_dt > stable_timestep(w, *params)) {
        g_last_error = "substep dt is not finite, not positive or above the CFL bound";
        return TMPM_ERR_INVALID_INPUT;
    }
    a->params = *params;
    a->dt = substep_dt;
    a->substeps = substeps;
    a->every = std::min(checkpoint_every, substeps);
    a->device = device;
    a->n = w.n;
    AdjParams &P = a->P;
    const double h = params->cell_width;
    P.h = static_cast<float>(h);
    P.inv_h = 1.0f / P.h;
    P.inv_d = static_cast<float>(4.0 / (h * h));
    P.dt = static_cast<float>(substep_dt);
    P.gx = static_cast<float>(params->gravity[0]);
    P.gy = static_cast<float>(params->gravity[1]);
    P.gz = static_cast<float>(params->gravity[2]);
    P.wall_mode = params->wall_mode;
    size_t nodes = 1;
    for (int k = 0; k < 3; ++k) {
        P.bmin[k] = static_cast<float>(params->bounds_min[k]);
        P.bmax[k] = static_cast<float>(params->bounds_max[k]);
        P.wall_lo[k] = wall_index_le(params->bounds_min[k] + h, h);
        P.wall_hi[k] = wall_index_ge(params->bounds_max[k] - h, h);
        int lo = static_cast<int>(std::floor(P.bmin[k] * P.inv_h - 0.5f)) - 1;
        int hi = static_cast<int>(std::floor(P.bmax[k] * P.inv_h - 0.5f)) + 3;
        P.lo[k] = lo;
        P.dim[k] = hi - lo + 1;
        nodes *= static_cast<size_t>(P.dim[k]);
    }
    if (nodes > (size_t(1) << 28)) {
        g_last_error = "domain too large for the dense node array";
        return TMPM_ERR_CAPACITY;
    }
    a->nodes = static_cast<int>(nodes);
    P.n = static_cast<int>(w.n);
    P.stride = w.n;
    const size_t n = w.n;
    HostVec<float> m(n), v(n), r(n), d(n), nu(n), S0(kRows * n);
    HostVec<uint8_t> fx(n);
    cudaError_t e;
    if ((e = cudaSetDevice(device))) {
        g_last_error = std::string("adjoint setup: ") + cudaGetErrorString(e);
        return TMPM_ERR_DEVICE;
    }
    a->whole_forward = n <= TmpmAdjoint::whole_room(k_rollout_forward<kRolloutThreads>);
    a->whole_backward = n <= std::min(whole_backward_particles(), TmpmAdjoint::whole_room(k_rollout_backward<kRolloutThreads>));
    a->order = rollout_order(w, P, kRolloutThreads);
    a->each_range([&](size_t begin, size_t end) {
        for (size_t j = begin; j < end; ++j) {
            const size_t i = a->order[j];
            m[j] = static_cast<float>(w.mass[i]);
            v[j] = static_cast<float>(w.vol[i]);
            r[j] = static_cast<float>(w.radius[i]);
            d[j] = static_cast<float>(w.damping[i]);
            nu[j] = static_cast<float>(w.mparams[5 * i + 1]);
            fx[j] = w.fixed[i];
            for (int k = 0; k < 3; ++k) {
                S0[k * n + j] = static_cast<float>(w.pos[3 * i + k]);
                S0[(3 + k) * n + j] = static_cast<float>(w.vel[3 * i + k]);
            }
            for (int k = 0; k < 9; ++k) {
                S0[(6 + k) * n + j] = static_cast<float>(w.C[9 * i + k]);
                S0[(15 + k) * n + j] = static_cast<float>(w.F[9 * i + k]);
            }
        }
    });
    const uint32_t segments = (substeps + a->every - 1) / a->every;
    const size_t sf = kRows * n;
    if ((e = cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking)) ||
        (e = cudaStreamCreateWithFlags(&a->side, cudaStreamNonBlocking)) ||
        (e = cudaEventCreateWithFlags(&a->ev_fork, cudaEventDisableTiming)) ||
        (e = cudaEventCreateWithFlags(&a->ev_replayed, cudaEventDisableTiming)) ||
        (e = cudaEventCreateWithFlags(&a->ev_swept, cudaEventDisableTiming)) ||
        (e = a->mass.alloc(n)) || (e = a->vol.alloc(n)) || (e = a->radius.alloc(n)) || (e = a->damping.alloc(n)) ||
        (e = a->nu.alloc(n)) || (e = a->initial.alloc(sf)) || (e = a->E.alloc(n)) || (e = a->Ebar.alloc(n)) || (e = a->fixed.alloc(n)) ||
        (e = a->ckpt.alloc(segments * sf)) || (e = a->adj[0].alloc(sf)) || (e = a->adj[1].alloc(sf)) ||
        (e = a->part.alloc(sf)) || (e = a->grid.alloc(nodes)) || (e = a->gv.alloc(nodes)) ||
        (e = a->gvb.alloc(nodes)) || (e = a->err.alloc(1)) || (e = a->gmb.alloc(nodes)) ||
        (e = a->bounds.alloc(6 * static_cast<size_t>(substeps) + 1))) {
        g_last_error = std::string("adjoint setup: ") + cudaGetErrorString(e);
        return TMPM_ERR_DEVICE;
    }
    for (int set = 0; set < 2; ++set)
        if ((e = a->seg[set].alloc(std::max<size_t>(a->every, 2) * sf)) ||
            (e = a->seg_grid[set].alloc(static_cast<size_t>(a->every) * nodes)) ||
            (e = a->seg_gv[set].alloc(static_cast<size_t>(a->every) * nodes)) ||
            (e = a->seg_R[set].alloc(a->every * 9 * n))) {
            g_last_error = std::string("adjoint setup: ") + cudaGetErrorString(e);
            return TMPM_ERR_DEVICE;
        }
    cudaMemcpyAsync(a->mass.ptr, m.data(), sizeof(float) * n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->vol.ptr, v.data(), sizeof(float) * n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->radius.ptr, r.data(), sizeof(float) * n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->damping.ptr, d.data(), sizeof(float) * n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->nu.ptr, nu.data(), sizeof(float) * n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->fixed.ptr, fx.data(), n, cudaMemcpyHostToDevice, a->stream);
    cudaMemcpyAsync(a->initial.ptr, S0.data(), sizeof(float) * S0.size(), cudaMemcpyHostToDevice, a->stream);
    if ((e = cudaStreamSynchronize(a->stream))) {
        g_last_error = std::string("adjoint setup: ") + cudaGetErrorString(e);
        return TMPM_ERR_DEVICE;
    }
    *out = a.release();
    return TMPM_OK;
}

void tmpm_adjoint_destroy(TmpmAdjoint *a) { delete a; }

size_t tmpm_adjoint_particle_count(const TmpmAdjoint *a) { return a ? a->n : 0; }

TmpmStatus tmpm_adjoint_forward(TmpmAdjoint *a, const double *velocity0, const double *young, double *position_out,
                                double *velocity_out) {
    if (!a) return TMPM_ERR_INVALID_INPUT;
    cudaSetDevice(a->device);
    a->have_forward = false;
    return a->forward(velocity0, young, position_out, velocity_out);
}

TmpmStatus tmpm_adjoint_backward(TmpmAdjoint *a, const double *position_grad, const double *velocity_grad,
                                 double *velocity0_grad, double *young_grad) {
    if (!a) return TMPM_ERR_INVALID_INPUT;
    cudaSetDevice(a->device);
    return a->backward(position_grad, velocity_grad, velocity0_grad, young_grad);
}

int32_t tmpm_debug_rollout_whole(const TmpmAdjoint *a) {
    return a ? (a->whole_forward ? 1 : 0) | (a->whole_backward ? 2 : 0) : 0;
}

void tmpm_debug_rollout_stepwise(TmpmAdjoint *a) {
    if (!a) return;
    cudaSetDevice(a->device);
    cudaStreamSynchronize(a->stream);
    if (a->fwd_exec) cudaGraphExecDestroy(a->fwd_exec);
    if (a->bwd_exec) cudaGraphExecDestroy(a->bwd_exec);
    a->fwd_exec = a->bwd_exec = nullptr;
    a->whole_forward = a->whole_backward = false;
}

const char *tmpm_adjoint_last_error_message(const TmpmAdjoint *a) {
    return a ? a->last_error.c_str() : g_last_error.c_str();
}

}  // extern "C"
