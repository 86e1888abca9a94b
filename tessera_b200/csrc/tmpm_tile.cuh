// tmpm_tile.cuh -- shared-memory tiles of grid nodes: index arithmetic, the
// fixed-point scale and the gather, for the transfer kernels and the
// differentiable rollout.
#pragma once

#include "tmpm_device.cuh"

namespace tmpm {

// Tile strides padded against shared-memory bank conflicts.  The 32 lanes of
// a warp hold particles of 32 neighbouring cells (with 8 per cell, a 2 x 4 x 4
// group in the chunk's cell Morton order, see lane_cell); with a y stride of
// 4 mod 8 and an x stride of 16 mod 32 their tile entries x * 16 + y * 4 + z
// are distinct mod 32, so a scatter atomic of the warp touches 32 banks and a
// gather load of a quarter-warp (a 1 x 2 x 4 slab) 8 distinct bank groups.
// Measured on the dam break: 2.24 -> 1.35 wavefronts per shared atomic.
__device__ __forceinline__ void tile_strides(int d1, int d2, int &s1, int &s2) {
    s2 = d2 + ((4 - d2) & 7);
    s1 = d1 * s2;
    s1 += (16 - s1) & 31;
}

// Split a padded tile index t (strides s1, s2) into (tx, ty, tz) without
// division, with a multiplier just above 2^22 / d (t / d = (t * m) >> 22) or, for
// a tile of more than 2304 entries, just above 2^32 / d (the high word of t * m).
// Exact for every tile index.  m d - 2^22 < 1.2 d + 1: the quotient is exact
// while t (1.2 d + 1) < 2^22, and a box has at least three x planes, so t < 2304
// and d <= 768 (t * m < 2^32 with d >= 3); the approximate reciprocal is off by
// less than the 0.1 added before truncation.  m d - 2^32 < 3200 + d: exact while
// t (3200 + d) < 2^32; the factor 1 + 2^-21 covers the reciprocal's two ulps.
template <bool WIDE>
__device__ __forceinline__ unsigned split_factor(int d) {
    if (WIDE) return static_cast<unsigned>(__fdividef(4294967296.0f, static_cast<float>(d)) * (1.0f + 4.76837158e-7f)) + 1u;
    return static_cast<unsigned>(__fdividef(4194304.0f, static_cast<float>(d)) + 0.1f) + 1u;
}
template <bool WIDE>
struct SplitP {
    int s1, s2;
    unsigned m1, m2;
    __device__ __forceinline__ SplitP(int s1_, int s2_)
        : s1(s1_), s2(s2_), m1(split_factor<WIDE>(s1_)), m2(split_factor<WIDE>(s2_)) {}
    static __device__ __forceinline__ int quotient(int t, unsigned m) {
        if (WIDE) return static_cast<int>(__umulhi(static_cast<unsigned>(t), m));
        return static_cast<int>((static_cast<unsigned>(t) * m) >> 22);
    }
    __device__ __forceinline__ void operator()(int t, int &tx, int &ty, int &tz) const {
        tx = quotient(t, m1);
        const int r = t - tx * s1;
        ty = quotient(r, m2);
        tz = r - ty * s2;
    }
};

// Largest power of two s with total * s <= 2^30 (exponent clamped to the normal
// range), from the exponent bits: total lies in (2^k, 2^(k+1)], s = 2^(29-k).
__device__ __forceinline__ float pow2_scale(float total) {
    const int k = (__float_as_int(fmaxf(total, 1e-30f)) - 1) >> 23;  // biased exponent of the largest float below total
    return __int_as_float(min(max(29 + 127 + 127 - k, 7), 247) << 23);
}
// 1 / s for a power of two s in the normal range.
__device__ __forceinline__ float pow2_inverse(float s) { return __int_as_float((254 << 23) - __float_as_int(s)); }

// A 3-vector as an (x, y) register pair, as a 16-byte shared load returns it, and z.
struct V2Z {
    float2 xy;
    float z;
    __device__ __forceinline__ V2Z(float2 xy_, float z_) : xy(xy_), z(z_) {}
    __device__ __forceinline__ explicit V2Z(const float4 &g) : xy(make_float2(g.x, g.y)), z(g.z) {}
    __device__ __forceinline__ V3f v3() const { return mk(xy.x, xy.y, z); }
};
__device__ __forceinline__ V2Z operator*(const V2Z &a, float s) { return V2Z(__fmul2_rn(make_float2(s, s), a.xy), s * a.z); }
__device__ __forceinline__ V2Z fma2z(float s, const V2Z &a, const V2Z &b) {
    return V2Z(__ffma2_rn(make_float2(s, s), a.xy, b.xy), fmaf(s, a.z, b.z));
}

// Sum_i w_i v_i (vs) and the first moments about the stencil's centre node
// (m0, m1, m2: sum_i w_i (offset - 1) v_i along x, y, z) of the x, y, z
// components, factored by axis: along z a row's sum r and moment d, over y a
// plane's sums, over x the particle's.  row(a, c) points at the three nodes of
// row (a, c).  With dpos = (offset - 1) h + (1 - f) h, sum_i w_i v_i dpos_i^T
// follows: 80 vector operations instead of 27 nodes x 4.  Rows are paired
// (Blackwell FFMA2 on the node's own register pair); pairing planes too costs
// weight pairs in registers (84 / 120 bytes of spills at 64 registers, 16 here).
// 64 substeps of the 4.05M-particle dam break: 22.97 ms, all scalar 23.14, all
// paired 23.94.
template <typename Row>
__device__ __forceinline__ void gather_moments(const float wx[3], const float wy[3], const float wz[3], Row row_at, V3f &vs,
                                               V3f &m0, V3f &m1, V3f &m2) {
    vs = m0 = m1 = m2 = mk(0, 0, 0);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        V3f s0 = mk(0, 0, 0), s1 = s0, s2 = s0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float4 *const row = row_at(a, c);
            const V2Z p0 = V2Z(row[0]) * wz[0], p2 = V2Z(row[2]) * wz[2];
            const V3f r = fma2z(wz[1], V2Z(row[1]), fma2z(1.0f, p0, p2)).v3();
            const V3f d = fma2z(-1.0f, p0, p2).v3();
            s0 = s0 + r * wy[c];
            if (c == 0) s1 = s1 - r * wy[0];
            if (c == 2) s1 = s1 + r * wy[2];
            s2 = s2 + d * wy[c];
        }
        vs = vs + s0 * wx[a];
        if (a == 0) m0 = m0 - s0 * wx[0];
        if (a == 2) m0 = m0 + s0 * wx[2];
        m1 = m1 + s1 * wx[a];
        m2 = m2 + s2 * wx[a];
    }
}

}  // namespace tmpm
