// tmpm_transfer.cuh -- the transfer kernels (P2G, fused G2P2G, G2P) and their launchers.
//
// Included by one translation unit per variant (tmpm_transfer_*.cu), so that
// the variants compile in parallel.
//
// Each CTA owns a chunk of consecutive particles in storage order (sorted by
// block and cell; 256 or 128 per chunk, the launch shape's CTA size, see
// kLaunchShapes; grid blocks of 4^3 or 8^3 cells, the template parameter BS).
// It stages the grid nodes its particles touch in a shared-memory
// box ("tile"): the gather tile holds step-n velocities, the scatter tile
// accumulates step-(n+1) mass and momentum with shared atomics and is flushed
// to the block pool with one float4 atomic per touched node.  Chunks whose box
// is too large (scattered particles) fall back to per-node global access.
//
// In a session the fused transfer of one scene runs as k_transfer_fast (the
// common path only) with k_transfer_deferred beside and after it for the
// chunks the common path does not cover (see transfer_chunk).
#pragma once

#include <algorithm>
#include <climits>

#include "tmpm_grid.cuh"
#include "tmpm_tile.cuh"

namespace tmpm {

namespace {

// Box edge in cells: only bounds the arithmetic (a padded entry count far
// inside int range); the entry and block counts decide whether a box fits.
// An elongated box (a chunk that wraps from one row of blocks to the next
// in storage order) fits when its volume does.
constexpr int kTileMaxDim = 64;
// Box nodes a CTA of `threads` particles stages: 9 per particle (2304 nodes,
// one 36 KB shared buffer, for 256; the most that keeps the static shared
// memory of the variants with the obstacle contact under 48 KB), used as the
// gather tile and then as the scatter tile.  Every transfer kernel stages the
// same box size, since a record one kernel writes is read by another.  On the
// evolved dam break 1.5 % of the chunks have boxes above 2048 entries and
// 1.0 % above 2304; those take the direct path (fused launch 0.428 -> 0.421 ms
// with the larger tile).
constexpr int tile_nodes(int threads) { return threads * 9; }
// A whole-segment kernel's chunks are alone with one or three others on their SM
// and share no record with another kernel, so its tile takes what shared memory
// is left: 22 nodes per particle (88 KB of dynamic shared memory for 256).  A
// chunk on the direct path (sorted particles that jump between blocks) holds up
// every barrier of the segment: 16 substeps of the 39,304-particle snow block
// 593 -> 472 us, of the 55k elastic block 406 -> 403 us, with the larger tile.
constexpr int segment_tile_nodes(int threads) { return threads * 22; }
// Blocks a box may span, by its tile's size.
constexpr int tile_blocks(int threads, int tile) { return tile > tile_nodes(threads) ? kCacheStride - 16 : 128; }
constexpr int kCacheHeader = 16;

struct Box {
    int lo[3];
    int dim[3];
    int blo[3];
    int nb[3];
    int nodes;  // tile entries: dim[0] * s1
    int nbt;
    int ok;
    uint32_t color;
    int s1, s2;  // tile strides of x and y (z: 1)
};

// Node index inside its block of edge 2^BS cells (x-major).
template <int BS>
__device__ __forceinline__ int node_local(int cx, int cy, int cz) {
    constexpr int m = (1 << BS) - 1;
    return ((cx & m) << (2 * BS)) | ((cy & m) << BS) | (cz & m);
}

// Split a row-major tile index t (dims d0 x d1 x d2, t < 2^20) into (tx, ty, tz)
// without integer division: (t + 0.5) / d lies at least 1 / (2 d) from an
// integer, far above the f32 error of (t + 0.5) * (1 / d), so truncation is exact.
struct Split3 {
    int d1, d2;
    float inv_d1, inv_d2;
    __device__ __forceinline__ Split3(int d1_, int d2_)
        : d1(d1_), d2(d2_), inv_d1(1.0f / static_cast<float>(d1_)), inv_d2(1.0f / static_cast<float>(d2_)) {}
    __device__ __forceinline__ void operator()(int t, int &tx, int &ty, int &tz) const {
        const int q = static_cast<int>((static_cast<float>(t) + 0.5f) * inv_d2);
        tz = t - q * d2;
        tx = static_cast<int>((static_cast<float>(q) + 0.5f) * inv_d1);
        ty = q - tx * d1;
    }
};

// Block-wide min/max of base cells and colours; thread 0 fills `box`.
template <int THREADS, int BS, int TILE>
__device__ __forceinline__ void reduce_box(bool valid, const int b[3], uint32_t color, int (*red)[8], Box &box) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int vals[8];
    for (int a = 0; a < 3; ++a) {
        vals[a] = valid ? b[a] : INT_MAX;
        vals[3 + a] = valid ? b[a] : INT_MIN;
    }
    vals[6] = valid ? static_cast<int>(color) : INT_MAX;
    vals[7] = valid ? static_cast<int>(color) : INT_MIN;
    int r[8];
    for (int a = 0; a < 3; ++a) r[a] = __reduce_min_sync(0xffffffffu, vals[a]);
    for (int a = 3; a < 6; ++a) r[a] = __reduce_max_sync(0xffffffffu, vals[a]);
    r[6] = __reduce_min_sync(0xffffffffu, vals[6]);
    r[7] = __reduce_max_sync(0xffffffffu, vals[7]);
    if (lane == 0)
        for (int a = 0; a < 8; ++a) red[warp][a] = r[a];
    __syncthreads();
    if (threadIdx.x == 0) {
        int m[8];
        for (int a = 0; a < 8; ++a) m[a] = red[0][a];
        for (int w = 1; w < THREADS / 32; ++w) {
            for (int a = 0; a < 3; ++a) m[a] = min(m[a], red[w][a]);
            for (int a = 3; a < 6; ++a) m[a] = max(m[a], red[w][a]);
            m[6] = min(m[6], red[w][6]);
            m[7] = max(m[7], red[w][7]);
        }
        bool any = m[0] <= m[3];
        int nodes = 1, nbt = 1;
        bool ok = any && m[6] == m[7];
        for (int a = 0; a < 3 && ok; ++a) {
            long long d = static_cast<long long>(m[3 + a]) - m[a] + 3;
            if (d > kTileMaxDim) ok = false;
        }
        if (ok) {
            for (int a = 0; a < 3; ++a) {
                box.lo[a] = m[a];
                box.dim[a] = m[3 + a] - m[a] + 3;
                box.blo[a] = m[a] >> BS;
                box.nb[a] = ((m[3 + a] + 2) >> BS) - box.blo[a] + 1;
                nodes *= box.dim[a];
                nbt *= box.nb[a];
            }
            int s1 = 0, s2 = 0;
            tile_strides(box.dim[1], box.dim[2], s1, s2);
            box.s1 = s1;
            box.s2 = s2;
            nodes = box.dim[0] * s1;
            ok = nodes <= TILE && nbt <= tile_blocks(THREADS, TILE);
        }
        box.nodes = nodes;
        box.nbt = nbt;
        box.ok = ok ? 1 : 0;
        box.color = static_cast<uint32_t>(m[6]);
    }
    __syncthreads();
}

// The box of base cells m[0..2] .. m[3..5] (m[0] > m[3]: no particle), 2 cells wider.
template <int THREADS, int BS, int TILE>
__device__ __forceinline__ void box_of(const int m[], bool one_color, uint32_t color, Box &box) {
    bool ok = m[0] <= m[3] && one_color;
    int nodes = m[0] <= m[3] ? 1 : 0, nbt = 1;  // nodes 0: no valid particle
    for (int a = 0; a < 3 && ok; ++a)
        if (static_cast<long long>(m[3 + a]) - m[a] + 3 > kTileMaxDim) ok = false;
    if (ok) {
        for (int a = 0; a < 3; ++a) {
            box.lo[a] = m[a];
            box.dim[a] = m[3 + a] - m[a] + 3;
            box.blo[a] = m[a] >> BS;
            box.nb[a] = ((m[3 + a] + 2) >> BS) - box.blo[a] + 1;
            nodes *= box.dim[a];
            nbt *= box.nb[a];
        }
        tile_strides(box.dim[1], box.dim[2], box.s1, box.s2);
        nodes = box.dim[0] * box.s1;
        ok = nodes <= TILE && nbt <= tile_blocks(THREADS, TILE);
    }
    box.nodes = nodes;
    box.nbt = nbt;
    box.ok = ok ? 1 : 0;
    box.color = color;
}

// Box of base cells and colours plus the sums and maxima of two non-negative
// floats over the CTA, with one barrier: each warp reduces its lanes and
// publishes a partial, then every warp combines the partials itself (no second
// barrier, no shared result).  The maxima are taken on the float bits, whose
// integer order is the value order for non-negative floats.
template <int THREADS, int BS, int TILE>
__device__ __forceinline__ void reduce_box_sums(bool valid, const int b[3], uint32_t color, float &sum_a, float &sum_b,
                                                float &max_a, float &max_b, int (*red)[8], float (*redf)[4],
                                                Box &box) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int r[8];
    for (int a = 0; a < 3; ++a) {
        r[a] = __reduce_min_sync(0xffffffffu, valid ? b[a] : INT_MAX);
        r[3 + a] = __reduce_max_sync(0xffffffffu, valid ? b[a] : INT_MIN);
    }
    r[6] = __reduce_min_sync(0xffffffffu, valid ? static_cast<int>(color) : INT_MAX);
    r[7] = __reduce_max_sync(0xffffffffu, valid ? static_cast<int>(color) : INT_MIN);
    float fa = sum_a, fb = sum_b;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        fa += __shfl_xor_sync(0xffffffffu, fa, off);
        fb += __shfl_xor_sync(0xffffffffu, fb, off);
    }
    const unsigned ma = __reduce_max_sync(0xffffffffu, __float_as_uint(max_a));
    const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(max_b));
    if (lane == 0) {
        for (int a = 0; a < 8; ++a) red[warp][a] = r[a];
        redf[warp][0] = fa;
        redf[warp][1] = fb;
        redf[warp][2] = __uint_as_float(ma);
        redf[warp][3] = __uint_as_float(mb);
    }
    __syncthreads();
    constexpr int kWarps = THREADS / 32;
    const bool mine = lane < kWarps;
    int m[8];
    for (int a = 0; a < 3; ++a) {
        m[a] = __reduce_min_sync(0xffffffffu, mine ? red[lane][a] : INT_MAX);
        m[3 + a] = __reduce_max_sync(0xffffffffu, mine ? red[lane][3 + a] : INT_MIN);
    }
    m[6] = __reduce_min_sync(0xffffffffu, mine ? red[lane][6] : INT_MAX);
    m[7] = __reduce_max_sync(0xffffffffu, mine ? red[lane][7] : INT_MIN);
    fa = mine ? redf[lane][0] : 0.0f;
    fb = mine ? redf[lane][1] : 0.0f;
    max_a = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(redf[lane][2]) : 0u));
    max_b = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(redf[lane][3]) : 0u));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        fa += __shfl_xor_sync(0xffffffffu, fa, off);
        fb += __shfl_xor_sync(0xffffffffu, fb, off);
    }
    sum_a = fa;
    sum_b = fb;
    box_of<THREADS, BS, TILE>(m, m[6] == m[7], static_cast<uint32_t>(m[6]), box);
}

// The same for a chunk whose gather used its record: the namespace is the
// recorded one for every particle and the mass bound is the recorded scale's, so
// six extremes and the momentum bound's sum and maximum remain.  Each warp adds
// its extremes to shared words (initialised by chunk_extremes_init before an
// earlier barrier) with native integer atomics, and every thread reads the
// totals: one pass of warp reductions instead of two, 13 instead of 40.
__device__ __forceinline__ void chunk_extremes_init(int *ext) {
    if (threadIdx.x < 8) ext[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : (threadIdx.x < 6 ? INT_MIN : 0);
}
template <int THREADS, int BS, int TILE>
__device__ __forceinline__ void reduce_box_recorded(bool valid, const int b[3], const Box &gbox, float &sum_p,
                                                    float &max_p, int *ext, float *psum, Box &box) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int r[6];
    for (int a = 0; a < 3; ++a) {
        r[a] = __reduce_min_sync(0xffffffffu, valid ? b[a] : INT_MAX);
        r[3 + a] = __reduce_max_sync(0xffffffffu, valid ? b[a] : INT_MIN);
    }
    const unsigned mp = __reduce_max_sync(0xffffffffu, __float_as_uint(max_p));
    float f = sum_p;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
    if (lane == 0) {
        for (int a = 0; a < 3; ++a) {
            atomicMin(ext + a, r[a]);
            atomicMax(ext + 3 + a, r[3 + a]);
        }
        atomicMax(reinterpret_cast<unsigned *>(ext) + 6, mp);
        psum[warp] = f;
    }
    __syncthreads();
    int m[6];
    for (int a = 0; a < 6; ++a) m[a] = ext[a];
    max_p = __uint_as_float(reinterpret_cast<const unsigned *>(ext)[6]);
    f = psum[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) f += psum[w];
    sum_p = f;
    box_of<THREADS, BS, TILE>(m, true, gbox.color, box);
}

// A CTA in which one particle's mass or momentum bound exceeds this share of
// the CTA's total scatters through the direct path (f32 global atomics per
// node, each node accurate relative to its own magnitude): its fixed-point
// scale would be set by that particle alone and would coarsen the quantum of
// every node its neighbours reach.
constexpr float kFloatModeShare = 1.0f / 8.0f;

__device__ __forceinline__ void quad_weights(float f, float w[3]) {
    w[0] = 0.5f * (1.5f - f) * (1.5f - f);
    w[1] = 0.75f - (f - 1.0f) * (f - 1.0f);
    w[2] = 0.5f * (f - 0.5f) * (f - 0.5f);
}

template <int BS>
__device__ __forceinline__ int tile_block_index(const Box &bx, int cx, int cy, int cz) {
    return (((cx >> BS) - bx.blo[0]) * bx.nb[1] + ((cy >> BS) - bx.blo[1])) * bx.nb[2] + ((cz >> BS) - bx.blo[2]);
}

// Component c of stored row i (byte offset 4 i, below 2^32): a base that is the
// same for every thread and one 32-bit offset per thread, instead of a 64-bit
// address computed per component.
__device__ __forceinline__ float load_row(const float *base, size_t cap, int c, uint32_t off) {
    return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(base + c * cap) + off);
}
__device__ __forceinline__ void store_row(float *base, size_t cap, int c, uint32_t off, float v) {
    *reinterpret_cast<float *>(reinterpret_cast<char *>(base + c * cap) + off) = v;
}
__device__ __forceinline__ V3f load_v3(const float *base, size_t cap, uint32_t off) {
    return mk(load_row(base, cap, 0, off), load_row(base, cap, 1, off), load_row(base, cap, 2, off));
}
__device__ __forceinline__ void store_v3(float *base, size_t cap, uint32_t off, V3f v) {
    store_row(base, cap, 0, off, v.x);
    store_row(base, cap, 1, off, v.y);
    store_row(base, cap, 2, off, v.z);
}
__device__ __forceinline__ M3f load_m3(const float *base, size_t cap, uint32_t off) {
    M3f m;
    m.c0 = mk(load_row(base, cap, 0, off), load_row(base, cap, 1, off), load_row(base, cap, 2, off));
    m.c1 = mk(load_row(base, cap, 3, off), load_row(base, cap, 4, off), load_row(base, cap, 5, off));
    m.c2 = mk(load_row(base, cap, 6, off), load_row(base, cap, 7, off), load_row(base, cap, 8, off));
    return m;
}
__device__ __forceinline__ void store_m3(float *base, size_t cap, uint32_t off, const M3f &m) {
    store_row(base, cap, 0, off, m.c0.x);
    store_row(base, cap, 1, off, m.c0.y);
    store_row(base, cap, 2, off, m.c0.z);
    store_row(base, cap, 3, off, m.c1.x);
    store_row(base, cap, 4, off, m.c1.y);
    store_row(base, cap, 5, off, m.c1.z);
    store_row(base, cap, 6, off, m.c2.x);
    store_row(base, cap, 7, off, m.c2.y);
    store_row(base, cap, 8, off, m.c2.z);
}

// F of stored row `off`; `isotropic`: a multiple of the identity whose first
// component alone is current.
__device__ __forceinline__ void load_deformation(const float *base, size_t cap, uint32_t off, bool isotropic, M3f &F) {
    if (isotropic) {
        const float s = load_row(base, cap, 0, off);
        F = M3f{mk(s, 0, 0), mk(0, s, 0), mk(0, 0, s)};
    } else {
        F = load_m3(base, cap, off);
    }
}

// The blocks a particle's 3 x 3 x 3 stencil reaches from base cell b: at most
// two per axis, slot (qx << 2) | (qy << 1) | qz for block (b >> BS) + q.  Each
// thread looks up (or, INSERT, finds or inserts) the distinct ones and stores
// the ids at ids[slot * THREADS], the unreached slots -1.
//
// Bound by latency: a CTA on this path is one of a few beside the fast kernel,
// and a lookup is a key load and then a value load.  So the first slot of every
// reached block is read at once, key and value together (one memory round trip
// instead of up to sixteen); only a block whose first slot holds another key,
// or whose id is not published yet, goes through the probing functions.  An id
// read here without acquire is safe to use: an id is written once, after its
// key, and the pools' nodes are zeroed before the table's first insert.
template <int THREADS, int BS, bool INSERT>
__device__ __forceinline__ void stencil_blocks(const GridTable &g, const int b[3], uint32_t ns, int *ids,
                                               uint32_t *status) {
    const int g0 = b[0] >> BS, g1 = b[1] >> BS, g2 = b[2] >> BS;
    const int e0 = ((b[0] + 2) >> BS) - g0, e1 = ((b[1] + 2) >> BS) - g1, e2 = ((b[2] + 2) >> BS) - g2;
    unsigned long long found[8];
    uint32_t val[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int qx = q >> 2, qy = (q >> 1) & 1, qz = q & 1;
        found[q] = kEmptyKey;
        val[q] = kPendingId;
        if (qx <= e0 && qy <= e1 && qz <= e2) {
            const uint32_t slot = hash_slot(block_key(g0 + qx, g1 + qy, g2 + qz, ns), g.mask);
            found[q] = __ldcg(g.keys + slot);
            val[q] = __ldcg(g.vals + slot);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int qx = q >> 2, qy = (q >> 1) & 1, qz = q & 1;
        const unsigned long long key = block_key(g0 + qx, g1 + qy, g2 + qz, ns);
        ids[q * THREADS] = found[q] == key && val[q] < kInvalidId ? static_cast<int>(val[q]) : -1;
    }
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        const int qx = q >> 2, qy = (q >> 1) & 1, qz = q & 1;
        if (qx > e0 || qy > e1 || qz > e2 || ids[q * THREADS] >= 0) continue;
        const unsigned long long key = block_key(g0 + qx, g1 + qy, g2 + qz, ns);
        if constexpr (INSERT)
            ids[q * THREADS] =
                find_or_insert_block(g, key, make_int4(g0 + qx, g1 + qy, g2 + qz, static_cast<int>(ns)), status);
        else
            ids[q * THREADS] = lookup_block(g, key);
    }
}
// The slot (stencil_blocks) of the block holding cell (cx, cy, cz) of the
// stencil based at b.
template <int BS>
__device__ __forceinline__ int stencil_block_slot(const int b[3], int cx, int cy, int cz) {
    return (((cx >> BS) - (b[0] >> BS)) << 2) | (((cy >> BS) - (b[1] >> BS)) << 1) | ((cz >> BS) - (b[2] >> BS));
}

// Shared memory of a transfer CTA, as pointers to its arrays.  One buffer
// holds the G2P gather tile (float4 per node) and then the P2G scatter tile
// (4 fixed-point ints per node, component-major).
template <int THREADS, bool OBST>
struct TransferSmem {
    float4 *tile;
    float (*fred)[4];
    int *blk;
    int *blk2;
    int *used;
    int (*red)[8];
    Box *box;
    Box *gbox;  // the G2P box, whose block ids the P2G reuses (shared: not held in registers)
    int *abort;
    int *record;   // a resident chunk's record (else in the cache array)
    int *ext;      // reduce_box_recorded
    float *psum;
    float (*park)[THREADS];  // the affine matrix across the obstacle contact
};
// The arrays, one set per kernel for each (THREADS, OBST): the deferred
// kernel's P2G-only and whole-chunk passes share them.
extern __shared__ float4 dynamic_tile[];  // of kernels whose tile exceeds tile_nodes (static shared memory ends at 48 KB)
template <int THREADS, bool OBST, int TILE>
__device__ __forceinline__ TransferSmem<THREADS, OBST> transfer_smem() {
    constexpr bool kDynamic = TILE > tile_nodes(THREADS);
    constexpr int kBlocks = tile_blocks(THREADS, TILE);
    __shared__ float4 static_tile[kDynamic ? 1 : TILE];
    float4 *const tile = kDynamic ? dynamic_tile : static_tile;
    __shared__ float fred[THREADS / 32][4];
    __shared__ int blk[kBlocks];
    __shared__ int blk2[kBlocks];
    __shared__ int used[kBlocks];
    __shared__ int red[THREADS / 32][8];
    __shared__ Box box;
    __shared__ Box gbox;
    __shared__ int abort_flag;
    __shared__ int record[kDynamic ? kCacheStride : 1];
    __shared__ __align__(16) int ext[8];
    __shared__ __align__(16) float psum[THREADS / 32];
    __shared__ float park[OBST ? 9 : 1][THREADS];
    return TransferSmem<THREADS, OBST>{tile, fred, blk, blk2, used, red, &box, &gbox, &abort_flag, record, ext, psum, park};
}

// Deferred-chunk lists (layout at DeferLists): 0 = P2G only, 1 = whole
// chunk, 2 + p = no record for a launch of step parity p.
__device__ __forceinline__ void defer_push(const SimParams &sp, int list, int chunk) {
    const uint32_t slot = atomicAdd(sp.defer + list, 1u);
    if (slot < static_cast<uint32_t>(sp.defer_cap))
        sp.defer[kDeferHeader + static_cast<size_t>(list) * sp.defer_cap + slot] = static_cast<uint32_t>(chunk);
}
// The tag of the per-CTA records that the P2G of a launch with this step
// index writes (1 or 2); a G2P accepts the tag of its own step index.  The
// general chunks of a fused transfer run beside the fast kernel and write
// their records meanwhile: the tag keeps the fast kernel from reading them
// as records of its own step.
__device__ __forceinline__ int record_tag(int step_index) { return 1 + (step_index & 1); }
// Added to the tag of a chunk whose particles are near an obstacle: the fast
// kernel would defer it whole, to run after it; with this bit the chunk is on the
// no-record list, and the general path runs it beside the fast kernel (with its
// record).  32 substeps of the 519k-particle dam break against a sphere, launch
// shape fixed: 2.15 -> 2.09 ms while the flow arrives, 2.53 -> 2.11 ms once it
// surrounds the sphere; 1.45M particles 4.81 -> 4.84 and 5.31 -> 4.94 ms.
constexpr int kRecordNear = 4;

#define TMPM_TRANSFER_PARAMS \
    ParticleSoA P, int n, const DevClass *__restrict__ classes, GridTable cur, GridTable next, SimParams sp, \
        const DevObstacle *__restrict__ obstacles, const float *__restrict__ planes, double *reactions, \
        uint32_t *status, int *__restrict__ cache
#define TMPM_TRANSFER_ARGS P, n, classes, cur, next, sp, obstacles, planes, reactions, status, cache

// One chunk of THREADS consecutive particles in storage order, by one CTA.
//
// FAST (the fused G2P2G of one scene without CPIC) compiles only the common
// path: the G2P box and block ids from the chunk's record, the gather from
// the tile and the fixed-point scatter tile.  A chunk without a record of
// this step is skipped (it is on the no-record list, which
// k_transfer_deferred runs beside the fast kernel); a chunk whose particles
// left the recorded box is deferred whole before any write; a chunk whose
// P2G box does not fit or has a dominant particle stores its particles'
// velocity and affine matrix and defers its P2G.  Without the fallback code
// (box reduction and hash lookups for the G2P, per-node global gathers and
// scatters) the fast kernel keeps the common path's values in registers: at
// 64 registers 24 / 28 bytes of spill stores / loads against 52 / 84 with the
// fallbacks compiled in.
//
// RESIDENT (whole-segment kernels: the CTA runs this chunk in every phase): the
// particle's position, F, plastic state and class word stay in `cs` and the
// chunk's record in shared memory from the opening P2G (which loads them) to
// the closing G2P (which stores them).
struct ChunkState {
    V3f x;
    M3f F;
    float pl[3];
    uint32_t cw, color;
    int kind;
};
template <int MODE, bool PLASTIC, int VARIANT, int THREADS, int BS, bool FAST, int TILE = tile_nodes(THREADS),
          bool RESIDENT = false>
__device__ __forceinline__ void transfer_chunk(TMPM_TRANSFER_PARAMS, const int chunk, const int step_index,
                                               const int apply_force, ChunkState *cs = nullptr) {
    constexpr bool MULTI = VARIANT == kMulti;
    constexpr bool CPIC = VARIANT == kCpic;
    constexpr bool OBST = has_obstacles(VARIANT);
    // The obstacle contact is compiled into the general path only: the fast
    // path tests each particle against the obstacles' reach (inline, no call)
    // and defers a chunk that may touch one.
    constexpr bool CONTACT = OBST && !FAST;
    static_assert(!FAST || (MODE == kModeG2P2G && !CPIC), "the fast path is the fused transfer without CPIC");
    constexpr int kTileNodes = TILE;
    constexpr bool kWideSplit = TILE > 2304;
    const TransferSmem<THREADS, CONTACT> S = transfer_smem<THREADS, CONTACT, TILE>();
    float4 *const s_gv = S.tile;
    int (*const s_sc)[kTileNodes] = reinterpret_cast<int (*)[kTileNodes]>(S.tile);
    float (*const s_fred)[4] = S.fred;
    int *const s_blk = S.blk;
    int *const s_blk2 = S.blk2;
    int *const s_used = S.used;
    int (*const s_red)[8] = S.red;
    Box &s_box = *S.box;
    Box &s_gbox = *S.gbox;
    int &s_abort = *S.abort;
    float (*const s_park)[THREADS] = S.park;

    const size_t cap = P.cap;
    const int i = chunk * THREADS + static_cast<int>(threadIdx.x);
    const uint32_t off = static_cast<uint32_t>(i) * 4u;
    const bool valid = i < n;
    int *const cc = RESIDENT ? S.record : cache + static_cast<size_t>(chunk) * kCacheStride;

    if (threadIdx.x == 0) s_abort = (*reinterpret_cast<volatile uint32_t *>(status) & kFatal) != 0;
    if (MODE != kModeG2P) {
        // The first barrier of the kernel orders these.
        if (MODE == kModeG2P2G) chunk_extremes_init(S.ext);
        for (int t = threadIdx.x; t < tile_blocks(THREADS, TILE); t += THREADS) s_used[t] = 0;
    }

    V3f x = mk(0, 0, 0);
    M3f F = m3_identity();
    uint32_t cw = 0;
    DevClass k;
    k.mass = 0.f;
    k.color = 0;
    if (RESIDENT && MODE != kModeP2G) {
        x = cs->x;
        cw = cs->cw;
        k.color = cs->color;
        k.kind = cs->kind;
    } else if (valid) {
        x = load_v3(P.x, cap, off);
        // all of a fluid's F between its first and last G2P of a segment; used
        // after the gather, loaded with x (a load there waits on DRAM: 22.8 ->
        // 22.6 ms for 64 substeps of the 4.05M-particle dam break)
        if (FAST) F.c0.x = load_row(P.F, cap, 0, off);
        cw = P.cls[i];
        // the namespace and kind now; the whole record after the gather (below)
        k.color = classes[cw & kClassMask].color;
        k.kind = classes[cw & kClassMask].kind;
    }
    const int scene = MULTI ? static_cast<int>(k.color >> kSceneShift) : 0;
    const SceneParams *const scn = sp.scenes + scene;
#define SCN(f) (MULTI ? scn->f : sp.s0.f)
    const float h = SCN(h), inv_h = SCN(inv_h), inv_d = SCN(inv_d), dt = SCN(dt);
    // g2p_on: the particle completes substep step_index here; p2g_on: it scatters for step_index + 1.
    bool g2p_on = valid, p2g_on = valid;
    if (MULTI && valid) {
        const int steps = scn->steps;
        const bool dead = (__ldcg(sp.scene_status + scene) & kStatusResident) != 0;
        g2p_on = !dead && step_index < steps;
        p2g_on = !dead && step_index + 1 < steps;
    }
    uint32_t *const resident_flag = MULTI ? sp.scene_status + scene : status;
    // grid namespace at the current positions (colour, and CPIC side masks when on)
    uint32_t ns = CPIC ? particle_namespace(k.color, 1, sp.num_obstacles, obstacles, x) : k.color;
    const bool fixed = (cw & kFixedBit) != 0;
    // A fluid's F is a multiple of the identity after its first G2P of the
    // segment (F <- cbrt(det F) I, below): between that G2P and its last one
    // only the first component is read and written.
    const bool fluid = valid && !fixed && k.kind == kMatFluid;
    const bool isotropic = fluid && (MODE == kModeP2G ? step_index >= 0 : step_index > 0);
    const bool plastic = PLASTIC && g2p_on && k.kind >= kMatSnow;
    float pl[3] = {1.0f, 0.0f, 0.0f};
    if (RESIDENT && MODE != kModeP2G) {
        if (PLASTIC)
            for (int q = 0; q < 3; ++q) pl[q] = cs->pl[q];
    } else if (plastic) {
        const V3f q = load_v3(P.pl, cap, off);
        pl[0] = q.x;
        pl[1] = q.y;
        pl[2] = q.z;
    }
    V3f v = mk(0, 0, 0);
    M3f Cm = m3_zero();
    bool recorded = false;  // the gather used the chunk's record (CTA-uniform)
    if (threadIdx.x == 0) s_gbox.ok = 0;

    if (MODE == kModeP2G) {
        if (valid) {
            load_deformation(P.F, cap, off, isotropic, F);
            k = classes[cw & kClassMask];
        }
        if (RESIDENT) *cs = ChunkState{x, F, {pl[0], pl[1], pl[2]}, cw, k.color, k.kind};
        if (p2g_on) {
            v = load_v3(P.v, cap, off);
            Cm = load_m3(P.C, cap, off);
        }
    } else {
        // ------------------------------------------------------------- G2P
        const int b[3] = {base_cell(x.x, inv_h), base_cell(x.y, inv_h), base_cell(x.z, inv_h)};
        // The previous P2G of this CTA recorded the box and block ids for these
        // very positions (ids are stable within a batch), so normally no box
        // reduction and no hash lookup is needed.  A record that does not
        // cover every particle sends the CTA through the general path.
        // The negative tag says that the P2G took the direct path: so does the
        // gather, without another box reduction.
        const int record = cc[0];
        bool use_cache = record == record_tag(step_index) ||
                         (CONTACT && record == (record_tag(step_index) | kRecordNear));
        if constexpr (FAST) {
            if (!use_cache) return;  // on the no-record list (CTA-uniform)
        }
        Box bx;
        for (int attempt = 0; attempt < (FAST ? 1 : 2); ++attempt) {
            if (use_cache) {
                bx.lo[0] = cc[8];
                bx.lo[1] = cc[9];
                bx.lo[2] = cc[10];
                bx.dim[0] = cc[11];
                bx.dim[1] = cc[12];
                bx.dim[2] = cc[13];
                bx.blo[0] = cc[1];
                bx.blo[1] = cc[2];
                bx.blo[2] = cc[3];
                bx.nb[0] = cc[4];
                bx.nb[1] = cc[5];
                bx.nb[2] = cc[6];
                bx.color = static_cast<uint32_t>(cc[7]);
                bx.nodes = cc[14];
                bx.nbt = bx.nb[0] * bx.nb[1] * bx.nb[2];
                bx.ok = 1;
                tile_strides(bx.dim[1], bx.dim[2], bx.s1, bx.s2);
            } else if (!FAST && record == -record_tag(step_index)) {
                bx.ok = 0;
                bx.color = 0;
            } else if constexpr (!FAST) {
                reduce_box<THREADS, BS, TILE>(g2p_on, b, ns, s_red, s_box);
                bx = s_box;
                if (bx.ok) {
                    const Split3 split(bx.nb[1], bx.nb[2]);
                    for (int t = threadIdx.x; t < bx.nbt; t += THREADS) {
                        int tx, ty, tz;
                        split(t, tx, ty, tz);
                        s_blk[t] = lookup_block(cur, block_key(bx.blo[0] + tx, bx.blo[1] + ty, bx.blo[2] + tz, bx.color));
                    }
                    __syncthreads();
                }
            }
            bool bad = use_cache && g2p_on &&
                       (b[0] < bx.lo[0] || b[1] < bx.lo[1] || b[2] < bx.lo[2] || b[0] + 2 >= bx.lo[0] + bx.dim[0] ||
                        b[1] + 2 >= bx.lo[1] + bx.dim[1] || b[2] + 2 >= bx.lo[2] + bx.dim[2] || ns != bx.color);
            if (bx.ok && !bad) {
                // four z-consecutive entries per step (the y stride is a multiple
                // of four): one index split for the four
                const SplitP<kWideSplit> split(bx.s1, bx.s2);
                for (int t = 4 * threadIdx.x; t < bx.nodes; t += 4 * THREADS) {
                    int tx, ty, tz;
                    split(t, tx, ty, tz);
                    if (ty >= bx.dim[1]) continue;  // padding
                    const int cx = bx.lo[0] + tx, cy = bx.lo[1] + ty;
                    const int tb0 = tile_block_index<BS>(bx, cx, cy, bx.blo[2] << BS);
                    const int local = node_local<BS>(cx, cy, 0);
                    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(s_gv + t));
                    int id = -1;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (tz + e >= bx.dim[2]) break;  // padding
                        const int cz = bx.lo[2] + tz + e;
                        if (e == 0 || (cz & ((1 << BS) - 1)) == 0) {
                            const int tb = tb0 + (cz >> BS) - bx.blo[2];
                            id = use_cache ? cc[kCacheHeader + tb] : s_blk[tb];
                            if (use_cache) s_blk[tb] = id;
                        }
                        if (id >= 0) {
                            // asynchronous 16-byte copy global -> shared (L2 only), no register staging
                            const float4 *src = cur.pool + (static_cast<size_t>(id) << (3 * BS)) +
                                                (local + (cz & ((1 << BS) - 1)));
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src) : "memory");
                        } else {
                            s_gv[t + e] = make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                    }
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            bad = __syncthreads_or(bad) != 0;
            if (!bad) break;
            if constexpr (FAST) {  // a particle left the recorded box: the whole chunk, nothing written yet
                if (threadIdx.x == 0) defer_push(sp, 1, chunk);
                return;
            }
            use_cache = false;
        }
        recorded = use_cache;
        if (s_abort) return;
        // the P2G below reuses the block ids of this box (read after its
        // barriers); published now, most of the box is dead through the gather
        if (MODE != kModeG2P && threadIdx.x == 0) s_gbox = bx;
        const V3f gp = mk(x.x * inv_h, x.y * inv_h, x.z * inv_h);
        const V3f fx = mk(gp.x - static_cast<float>(b[0]), gp.y - static_cast<float>(b[1]), gp.z - static_cast<float>(b[2]));
        float wx[3], wy[3], wz[3];
        quad_weights(fx.x, wx);
        quad_weights(fx.y, wy);
        quad_weights(fx.z, wz);
        V3f vel = mk(0, 0, 0);
        M3f aff = m3_zero();
        if (g2p_on && !fixed) {
            if (FAST || bx.ok) {
                const int t0 = (b[0] - bx.lo[0]) * bx.s1 + (b[1] - bx.lo[1]) * bx.s2 + (b[2] - bx.lo[2]);
                V3f vs, m0, m1, m2;
                gather_moments(wx, wy, wz, [&](int a, int c) { return s_gv + (t0 + a * bx.s1 + c * bx.s2); }, vs, m0, m1, m2);
                const float hd = h * inv_d;
                vel = vs;
                aff.c0 = (m0 + vs * (1.0f - fx.x)) * hd;
                aff.c1 = (m1 + vs * (1.0f - fx.y)) * hd;
                aff.c2 = (m2 + vs * (1.0f - fx.z)) * hd;
            } else {
                // Per-node global gather.  The stencil's blocks are looked up
                // first (the tile is unused on this path and holds each
                // thread's ids), so no node load waits on a lookup.
                float dxs[3], dys[3], dzs[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    dxs[a] = (a - fx.x) * h * inv_d;
                    dys[a] = (a - fx.y) * h * inv_d;
                    dzs[a] = (a - fx.z) * h * inv_d;
                }
                int *const ids = reinterpret_cast<int *>(s_gv) + threadIdx.x;
                stencil_blocks<THREADS, BS, false>(cur, b, ns, ids, status);
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int e = 0; e < 3; ++e) {
                            const int cx = b[0] + a, cy = b[1] + c, cz = b[2] + e;
                            const int id = ids[stencil_block_slot<BS>(b, cx, cy, cz) * THREADS];
                            float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (id >= 0)
                                val = __ldcg(cur.pool + static_cast<size_t>(id) * (1 << (3 * BS)) + node_local<BS>(cx, cy, cz));
                            const float w = wx[a] * wy[c] * wz[e];
                            const V3f nv = mk(val.x, val.y, val.z);
                            vel = vel + nv * w;
                            aff.c0 = aff.c0 + nv * (dxs[a] * w);
                            aff.c1 = aff.c1 + nv * (dys[c] * w);
                            aff.c2 = aff.c2 + nv * (dzs[e] * w);
                        }
            }
        }

        // F is read only now: it is not needed during the gather, whose
        // accumulators and weights are the kernel's peak register demand.  With
        // the obstacle contact (an out-of-line call, around which everything
        // live is saved) an updating particle reads F after the contact.
        const bool updates = g2p_on && !fixed;
        if (valid) {
            if (RESIDENT) F = cs->F;
            else if (FAST && isotropic) F = M3f{mk(F.c0.x, 0, 0), mk(0, F.c0.x, 0), mk(0, 0, F.c0.x)};
            else if (!CONTACT || !updates) load_deformation(P.F, cap, off, isotropic, F);
            k = classes[cw & kClassMask];
        }
        V3f pos = x;
        if (updates) {
            // Particle update (gpu.wgsl:885-1003; world.rs:443-463).
            if (apply_force) {
                const size_t w = P.widx[i], fs = P.force_stride;
                V3f f = mk(P.force[w], P.force[fs + w], P.force[2 * fs + w]);
                vel = vel + mk(f.x / k.mass, f.y / k.mass, f.z / k.mass) * dt;  // force / mass * dt (gpu.wgsl:885)
            }
            vel = vel * expf(-k.damping * dt);
            pos = x + vel * dt;
            const float radius = k.radius;
            if (SCN(has_bounds)) {
                for (int a = 0; a < 3; ++a) {
                    float lower = SCN(bmin[a]) + radius, upper = SCN(bmax[a]) - radius;
                    float pa = comp(pos, a), va = comp(vel, a);
                    if (pa < lower) {
                        set_comp(pos, a, lower);
                        set_comp(vel, a, fmaxf(va, 0.0f));
                    } else if (pa > upper) {
                        set_comp(pos, a, upper);
                        set_comp(vel, a, fminf(va, 0.0f));
                    }
                }
            }
            if constexpr (CONTACT) {
                // The surface function is an out-of-line call, around which
                // every live value is saved: the affine matrix waits in shared
                // memory and the class record is dropped (reloaded below), so
                // that only the position, velocity, radius and mass live across.
                const float pmass = k.mass;
                s_park[0][threadIdx.x] = aff.c0.x;
                s_park[1][threadIdx.x] = aff.c0.y;
                s_park[2][threadIdx.x] = aff.c0.z;
                s_park[3][threadIdx.x] = aff.c1.x;
                s_park[4][threadIdx.x] = aff.c1.y;
                s_park[5][threadIdx.x] = aff.c1.z;
                s_park[6][threadIdx.x] = aff.c2.x;
                s_park[7][threadIdx.x] = aff.c2.y;
                s_park[8][threadIdx.x] = aff.c2.z;
                for (int oi = 0; oi < sp.num_obstacles; ++oi) {
                    const DevObstacle &o = obstacles[oi];
                    if (!obstacle_may_contact(o, pos, radius)) continue;
                    V3f nrm;
                    float d = obstacle_surface(o, planes, pos, nrm);
                    if (d < radius) {
                        pos = pos + nrm * (radius - d);
                        V3f before = vel;
                        vel = contact_velocity(o, pos, vel, nrm);
                        if (sp.reactions)
                            add_reaction(reactions, oi, mk(o.center[0], o.center[1], o.center[2]), pos - nrm * radius,
                                         (before - vel) * pmass);
                    }
                }
                aff.c0 = mk(s_park[0][threadIdx.x], s_park[1][threadIdx.x], s_park[2][threadIdx.x]);
                aff.c1 = mk(s_park[3][threadIdx.x], s_park[4][threadIdx.x], s_park[5][threadIdx.x]);
                aff.c2 = mk(s_park[6][threadIdx.x], s_park[7][threadIdx.x], s_park[8][threadIdx.x]);
                k = classes[cw & kClassMask];
            }
        }
        if constexpr (OBST && FAST) {
            // A chunk in which some particle may touch an obstacle runs whole
            // through the general path, which has the contact: deferred here,
            // before this kernel writes anything or flags a failure for it.
            // The reach test is conservative (f32 rounding margins in the
            // reach and 5 % of a cell here), so a chunk that stays has no
            // contact, exactly as the general path would find.
            bool near = false;
            if (updates) {
                const float r = k.radius * 1.0001f + 0.05f * h;
                for (int oi = 0; oi < sp.num_obstacles; ++oi) near = near || obstacle_near(obstacles[oi], pos, r);
            }
            if (__syncthreads_or(near)) {
                if (threadIdx.x == 0) defer_push(sp, 1, chunk);
                return;
            }
        }
        if (updates) {
            if (CONTACT) {
                if (RESIDENT) F = cs->F;
                else load_deformation(P.F, cap, off, isotropic, F);
            }
            const M3f grad = add(m3_identity(), scale(aff, dt));  // F <- (I + dt C) F
            M3f Fn;
            bool plastic_ok = true;
            if (k.kind == kMatFluid) {
                // cbrt(det((I + dt C) F)) I; the determinant is the product of the factors'
                const float jf = isotropic ? F.c0.x * (F.c0.x * F.c0.x) : det(F);
                Fn = scale(m3_identity(), cbrtf(fmaxf(det(grad) * jf, 1e-9f)));
            } else {
                Fn = mul(grad, F);
                if (PLASTIC && k.kind >= kMatSnow) plastic_ok = project_plastic(k, Fn, pl);
            }
            // Resident failure detection (gpu.wgsl:946-994).
            bool failed = !finite3(pos) || !finite3(vel) || !finite_m(aff) || !finite_m(Fn);
            const float cx = __fsub_rn(__fmul_rn(pos.x, inv_h), 0.5f), cy = __fsub_rn(__fmul_rn(pos.y, inv_h), 0.5f),
                        cz = __fsub_rn(__fmul_rn(pos.z, inv_h), 0.5f);
            // floor(c) within [-131000, 131000]
            bool representable = cx >= -131000.0f && cx < 131001.0f && cy >= -131000.0f && cy < 131001.0f &&
                                 cz >= -131000.0f && cz < 131001.0f;
            failed = failed || !representable;
            if (!failed && SCN(has_bounds)) {
                // the base cells of the P2G below
                int nb3[3] = {__float2int_rd(cx), __float2int_rd(cy), __float2int_rd(cz)};
                for (int a = 0; a < 3; ++a)
                    failed = failed || nb3[a] < SCN(first_base[a]) || nb3[a] > SCN(last_base[a]);
            }
            if (sp.resident_checks) {
                if (k.kind == kMatCorotated || k.kind == kMatSnow || k.kind == kMatSand)
                    failed = failed || !regular_corotated(Fn);
                if (k.kind == kMatSandNeoHookean) {  // CFL with the elastic volume (gpu.wgsl:983-987)
                    float wave = k.wave * sqrtf(fmaxf(det(Fn), 1e-6f));
                    failed = failed || dt * fmaxf(wave, len(vel)) > 0.5f * h * (1.0f + 1e-4f);
                } else {
                    failed = failed || dt * (k.wave + len(vel)) > 0.4f * h * (1.0f + 1e-4f);
                }
                failed = failed || !plastic_ok;
                if (failed) atomicOr(resident_flag, kStatusResident);
            } else {
                if (finite3(pos) && !representable) atomicOr(status, kStatusCapacity);  // beyond the key range
                // no CPU fallback on this path: an unprojectable plastic state is unavailable here
                if (!plastic_ok) atomicOr(resident_flag, kStatusResident);
            }
            x = pos;
            v = vel;
            Cm = aff;
            F = Fn;
        }
        const bool last = MODE == kModeG2P || (MULTI && !p2g_on);
        if (RESIDENT && MODE != kModeG2P) {
            cs->x = x;
            cs->F = F;
            if (PLASTIC)
                for (int q = 0; q < 3; ++q) cs->pl[q] = pl[q];
        }
        if (g2p_on && (!RESIDENT || last)) {
            store_v3(P.x, cap, off, x);
            if (!fixed) {
                if (fluid && step_index > 0 && !last) store_row(P.F, cap, 0, off, F.c0.x);
                else store_m3(P.F, cap, off, F);
            }
            if (plastic && !fixed) store_v3(P.pl, cap, off, mk(pl[0], pl[1], pl[2]));
            // the last substep of the batch (per scene in a multi-scene batch) writes v and C back
            if (last) {
                store_v3(P.v, cap, off, v);
                store_m3(P.C, cap, off, Cm);
            }
        }
        if (MODE == kModeG2P) return;
    }

    // ----------------------------------------------------------------- P2G
    const int b[3] = {base_cell(x.x, inv_h), base_cell(x.y, inv_h), base_cell(x.z, inv_h)};
    const bool in_range =
        block_representable(b[0] >> BS, b[1] >> BS, b[2] >> BS) &&
        block_representable((b[0] + 2) >> BS, (b[1] + 2) >> BS, (b[2] + 2) >> BS);
    const bool active = p2g_on && in_range;
    if (p2g_on && !in_range) {
        if (sp.resident_checks) atomicOr(resident_flag, kStatusResident);
        else atomicOr(status, kStatusCapacity);
    }
    const V3f gp = mk(x.x * inv_h, x.y * inv_h, x.z * inv_h);
    const V3f fx = mk(gp.x - static_cast<float>(b[0]), gp.y - static_cast<float>(b[1]), gp.z - static_cast<float>(b[2]));
    float wx[3], wy[3], wz[3];
    quad_weights(fx.x, wx);
    quad_weights(fx.y, wy);
    quad_weights(fx.z, wz);
    M3f A = m3_zero();
    V3f mv = mk(0, 0, 0);
    float bound_m = 0.f, bound_p = 0.f;
    if (active) {
        M3f S = scaled_stress<!CONTACT && !PLASTIC>(k, F, Cm, -dt * inv_d, pl[0]);
        A = add(S, scale(Cm, k.mass));
        mv = v * k.mass;
        // |(m v + A dpos)_i| <= |m v_i| + 1.5 h sum_j |A_ij| and a particle's 27 weights sum to one,
        // so the chunk's sums bound every node value it produces.
        float r0 = fabsf(A.c0.x) + fabsf(A.c1.x) + fabsf(A.c2.x);
        float r1 = fabsf(A.c0.y) + fabsf(A.c1.y) + fabsf(A.c2.y);
        float r2 = fabsf(A.c0.z) + fabsf(A.c1.z) + fabsf(A.c2.z);
        bound_m = k.mass;
        bound_p = fmaxf(fmaxf(fabsf(mv.x) + 1.5f * h * r0, fabsf(mv.y) + 1.5f * h * r1), fabsf(mv.z) + 1.5f * h * r2);
        if (!(bound_p < 1e30f)) bound_p = 1e30f;  // non-finite state is flagged by the G2P checks
    }
    // the CTA's box and the sums of the bounds, with one barrier
    if (MODE != kModeP2G && CPIC) ns = particle_namespace(k.color, 1, sp.num_obstacles, obstacles, x);
    float tot_p = bound_p, max_p = bound_p, sm;
    Box bx;
    if (FAST || (MODE == kModeG2P2G && !CPIC && recorded)) {
        // the record's P2G summed the masses of these particles (or of a
        // superset that bounds them) and found none dominant
        sm = __int_as_float(cc[15]);
        reduce_box_recorded<THREADS, BS, TILE>(active, b, s_gbox, tot_p, max_p, S.ext, S.psum, bx);
    } else {
        float tot_m = bound_m, max_m = bound_m;
        reduce_box_sums<THREADS, BS, TILE>(active, b, ns, tot_m, tot_p, max_m, max_p, s_red, s_fred, bx);
        sm = pow2_scale(tot_m);
        if (max_m > tot_m * kFloatModeShare) bx.ok = 0;
    }
    if (MODE == kModeP2G && s_abort) return;
    // one dominant particle: the whole CTA takes the f32 direct path (CTA-uniform)
    if (max_p > tot_p * kFloatModeShare) bx.ok = 0;
    if constexpr (FAST) {
        if (!bx.ok) {
            // A chunk with nothing to scatter (every particle's scene is past
            // its last substep of the batch) needs no P2G and no record.
            if (bx.nodes == 0) {
                if (threadIdx.x == 0) cc[0] = 0;
                return;
            }
            // the P2G-only pass reads velocity and affine matrix from the
            // particle arrays (position, F and plastic state are stored)
            if (p2g_on) {
                store_v3(P.v, cap, off, v);
                store_m3(P.C, cap, off, Cm);
            }
            if (threadIdx.x == 0) defer_push(sp, 0, chunk);
            return;
        }
    }
    // A chunk that may touch an obstacle in the next substep, a quarter cell away
    // at most (CTA-uniform).
    bool near = false;
    if constexpr (CONTACT && !CPIC) {
        if (bx.ok && sp.defer && sp.num_obstacles > 0) {
            if (active) {
                const float r = k.radius * 1.0001f + 0.25f * h;
                for (int oi = 0; oi < sp.num_obstacles; ++oi) near = near || obstacle_near(obstacles[oi], x, r);
            }
            near = __syncthreads_or(near) != 0;
        }
    }
    if (bx.ok) {
        // every warp has finished its gather (barrier above): the buffer becomes the scatter tile
        // (a multiple of 16 entries: the x stride is)
        for (int t = 4 * threadIdx.x; t < bx.nodes; t += 4 * THREADS)
#pragma unroll
            for (int c = 0; c < 4; ++c) *reinterpret_cast<int4 *>(&s_sc[c][t]) = make_int4(0, 0, 0, 0);
        __syncthreads();
        // Shared accumulation in 32-bit fixed point: integer shared atomics are
        // native, float ones are not.  Power-of-two scales from the chunk bounds
        // keep every node sum below 2^30 (no overflow) with unbiased rounding.
        const float spv = pow2_scale(tot_p);
        if (active) {
            const int ox = b[0] - bx.lo[0], oy = b[1] - bx.lo[1], oz = b[2] - bx.lo[2];
            const float msc = k.mass * sm;
            float dxs[3], dys[3], dzs[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                dxs[a] = (a - fx.x) * h;
                dys[a] = (a - fx.y) * h;
                dzs[a] = (a - fx.z) * h;
            }
            // Paired f32 arithmetic: per node (m w s_m, w s_p) from (w_ac, w_ac) x (w_z m s_m, w_z s_p),
            // and the momentum's (x, y) pair.
            float2 zs[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) zs[e] = make_float2(wz[e] * msc, wz[e] * spv);
            const float2 c2xy = make_float2(A.c2.x, A.c2.y);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const V3f qa = mv + A.c0 * dxs[a];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const V3f qac = qa + A.c1 * dys[c];
                    const float wac = wx[a] * wy[c];
                    const float2 wac2 = make_float2(wac, wac);
                    const float2 qacxy = make_float2(qac.x, qac.y);
                    const int row = (ox + a) * bx.s1 + (oy + c) * bx.s2 + oz;
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        const float2 qxy = __ffma2_rn(c2xy, make_float2(dzs[e], dzs[e]), qacxy);
                        const float qz = qac.z + A.c2.z * dzs[e];
                        const float2 mw = __fmul2_rn(wac2, zs[e]);  // (w m s_m, w s_p)
                        const float2 pxy = __fmul2_rn(qxy, make_float2(mw.y, mw.y));
                        const int t = row + e;
                        atomicAdd(reinterpret_cast<unsigned *>(&s_sc[0][t]), static_cast<unsigned>(__float2int_rn(mw.x)));
                        atomicAdd(reinterpret_cast<unsigned *>(&s_sc[1][t]), static_cast<unsigned>(__float2int_rn(pxy.x)));
                        atomicAdd(reinterpret_cast<unsigned *>(&s_sc[2][t]), static_cast<unsigned>(__float2int_rn(pxy.y)));
                        atomicAdd(reinterpret_cast<unsigned *>(&s_sc[3][t]), static_cast<unsigned>(__float2int_rn(qz * mw.y)));
                    }
                }
            }
            // mark the (at most 8) blocks this particle's stencil touches
            const int bx0 = (b[0] >> BS) - bx.blo[0], bx1 = ((b[0] + 2) >> BS) - bx.blo[0];
            const int by0 = (b[1] >> BS) - bx.blo[1], by1 = ((b[1] + 2) >> BS) - bx.blo[1];
            const int bz0 = (b[2] >> BS) - bx.blo[2], bz1 = ((b[2] + 2) >> BS) - bx.blo[2];
            s_used[(bx0 * bx.nb[1] + by0) * bx.nb[2] + bz0] = 1;
            s_used[(bx0 * bx.nb[1] + by0) * bx.nb[2] + bz1] = 1;
            s_used[(bx0 * bx.nb[1] + by1) * bx.nb[2] + bz0] = 1;
            s_used[(bx0 * bx.nb[1] + by1) * bx.nb[2] + bz1] = 1;
            s_used[(bx1 * bx.nb[1] + by0) * bx.nb[2] + bz0] = 1;
            s_used[(bx1 * bx.nb[1] + by0) * bx.nb[2] + bz1] = 1;
            s_used[(bx1 * bx.nb[1] + by1) * bx.nb[2] + bz0] = 1;
            s_used[(bx1 * bx.nb[1] + by1) * bx.nb[2] + bz1] = 1;
        }
        __syncthreads();
        const Split3 split_b(bx.nb[1], bx.nb[2]);
        for (int t = threadIdx.x; t < bx.nbt; t += THREADS) {
            int id = -1;
            if (s_used[t]) {
                int tx, ty, tz;
                split_b(t, tx, ty, tz);
                int gx = bx.blo[0] + tx, gy = bx.blo[1] + ty, gz = bx.blo[2] + tz;
                // reuse the id the G2P box already holds for this block (same table)
                if (s_gbox.ok && s_gbox.color == bx.color) {
                    int rx = gx - s_gbox.blo[0], ry = gy - s_gbox.blo[1], rz = gz - s_gbox.blo[2];
                    if (rx >= 0 && ry >= 0 && rz >= 0 && rx < s_gbox.nb[0] && ry < s_gbox.nb[1] && rz < s_gbox.nb[2])
                        id = s_blk[(rx * s_gbox.nb[1] + ry) * s_gbox.nb[2] + rz];
                }
                if (id < 0)
                    id = find_or_insert_block(next, block_key(gx, gy, gz, bx.color),
                                              make_int4(gx, gy, gz, static_cast<int>(bx.color)), status);
            }
            s_blk2[t] = id;
            cc[kCacheHeader + t] = id;
        }
        if (threadIdx.x == 0) {
            cc[0] = record_tag(step_index + 1) | (near ? kRecordNear : 0);
            if (near) defer_push(sp, 2 + ((step_index + 1) & 1), chunk);
            cc[1] = bx.blo[0];
            cc[2] = bx.blo[1];
            cc[3] = bx.blo[2];
            cc[4] = bx.nb[0];
            cc[5] = bx.nb[1];
            cc[6] = bx.nb[2];
            cc[7] = static_cast<int>(bx.color);
            cc[8] = bx.lo[0];
            cc[9] = bx.lo[1];
            cc[10] = bx.lo[2];
            cc[11] = bx.dim[0];
            cc[12] = bx.dim[1];
            cc[13] = bx.dim[2];
            cc[14] = bx.nodes;
            cc[15] = __float_as_int(sm);
        }
        __syncthreads();
        const float inv_sm = pow2_inverse(sm), inv_sp = pow2_inverse(spv);
        const SplitP<kWideSplit> split_n(bx.s1, bx.s2);
        for (int t = 4 * threadIdx.x; t < bx.nodes; t += 4 * THREADS) {  // four entries per step, as the fill
            const int4 m = *reinterpret_cast<const int4 *>(&s_sc[0][t]), px = *reinterpret_cast<const int4 *>(&s_sc[1][t]),
                       py = *reinterpret_cast<const int4 *>(&s_sc[2][t]), pz = *reinterpret_cast<const int4 *>(&s_sc[3][t]);
            const int any[4] = {m.x | px.x | py.x | pz.x, m.y | px.y | py.y | pz.y, m.z | px.z | py.z | pz.z,
                                m.w | px.w | py.w | pz.w};
            if ((any[0] | any[1] | any[2] | any[3]) == 0) continue;
            int tx, ty, tz;
            split_n(t, tx, ty, tz);
            if (ty >= bx.dim[1]) continue;  // padding (zero by construction; never flushed)
            const int cx = bx.lo[0] + tx, cy = bx.lo[1] + ty;
            const int tb0 = tile_block_index<BS>(bx, cx, cy, bx.blo[2] << BS);
            const int local = node_local<BS>(cx, cy, 0);
            const int ms[4] = {m.x, m.y, m.z, m.w}, xs[4] = {px.x, px.y, px.z, px.w}, ys[4] = {py.x, py.y, py.z, py.w},
                      zs[4] = {pz.x, pz.y, pz.z, pz.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (any[e] == 0 || tz + e >= bx.dim[2]) continue;
                const int cz = bx.lo[2] + tz + e;
                const int id = s_blk2[tb0 + (cz >> BS) - bx.blo[2]];
                if (id < 0) continue;
                atomicAdd(next.pool + (static_cast<size_t>(id) << (3 * BS)) + (local + (cz & ((1 << BS) - 1))),
                          make_float4(static_cast<float>(ms[e]) * inv_sm, static_cast<float>(xs[e]) * inv_sp,
                                      static_cast<float>(ys[e]) * inv_sp, static_cast<float>(zs[e]) * inv_sp));
            }
        }
    } else {
        if (threadIdx.x == 0) {
            cc[0] = -record_tag(step_index + 1);
            if (sp.defer) defer_push(sp, 2 + ((step_index + 1) & 1), chunk);
        }
        if (active) {
            // Per-node global scatter, the stencil's blocks found or inserted
            // first (the tile is unused on this path: every warp is past its
            // gather, the barrier of the box reduction orders it).
            int *const ids = reinterpret_cast<int *>(s_gv) + threadIdx.x;
            stencil_blocks<THREADS, BS, true>(next, b, ns, ids, status);
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        const int cx = b[0] + a, cy = b[1] + c, cz = b[2] + e;
                        const int id = ids[stencil_block_slot<BS>(b, cx, cy, cz) * THREADS];
                        if (id < 0) continue;
                        float w = wx[a] * wy[c] * wz[e];
                        V3f dpos = mk((a - fx.x) * h, (c - fx.y) * h, (e - fx.z) * h);
                        V3f mom = (mv + mul(A, dpos)) * w;
                        atomicAdd(next.pool + static_cast<size_t>(id) * (1 << (3 * BS)) + node_local<BS>(cx, cy, cz),
                                  make_float4(w * k.mass, mom.x, mom.y, mom.z));
                    }
        }
    }
#undef SCN
}

// The general transfer: every chunk, one CTA each.
template <int MODE, bool PLASTIC, int VARIANT, int THREADS, int MINB, int BS>
__global__ void __launch_bounds__(THREADS, MINB) k_transfer(TMPM_TRANSFER_PARAMS) {
    transfer_chunk<MODE, PLASTIC, VARIANT, THREADS, BS, false>(TMPM_TRANSFER_ARGS, blockIdx.x, sp.step_index, sp.apply_force);
}

// The fast fused transfer: every chunk with a record of this step.
template <bool PLASTIC, int VARIANT, int THREADS, int MINB, int BS>
__global__ void __launch_bounds__(THREADS, MINB) k_transfer_fast(TMPM_TRANSFER_PARAMS) {
    transfer_chunk<kModeG2P2G, PLASTIC, VARIANT, THREADS, BS, true>(TMPM_TRANSFER_ARGS, blockIdx.x, sp.step_index, sp.apply_force);
}

// The deferred chunks of a fast fused transfer through the general path, a
// grid-stride loop of CTAs over a list.  PRE: the chunks without a record of
// this step (written by the previous launch's general P2Gs), run beside the
// fast kernel; otherwise the chunks the fast kernel deferred: P2G only, then
// whole chunks.  The register bound is the general kernel's: a CTA of this
// kernel running beside the fast kernel then takes one CTA slot of an SM, not
// the whole register file.
template <bool PRE, bool PLASTIC, int VARIANT, int THREADS, int BS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? TMPM_TRANSFER_MIN_BLOCKS : 8)
    k_transfer_deferred(TMPM_TRANSFER_PARAMS) {
    const uint32_t cap = static_cast<uint32_t>(sp.defer_cap);
    const uint32_t *const lists = sp.defer + kDeferHeader;
    if (PRE) {
        const int list = 2 + (sp.step_index & 1);
        const uint32_t count = min(sp.defer[list], cap);
        for (uint32_t e = blockIdx.x; e < count; e += gridDim.x) {
            __syncthreads();  // the previous chunk's last reads of shared memory
            transfer_chunk<kModeG2P2G, PLASTIC, VARIANT, THREADS, BS, false>(
                TMPM_TRANSFER_ARGS, static_cast<int>(lists[list * cap + e]), sp.step_index, sp.apply_force);
        }
    } else {
        const uint32_t np = min(sp.defer[0], cap), nw = min(sp.defer[1], cap);
        for (uint32_t e = blockIdx.x; e < np + nw; e += gridDim.x) {
            __syncthreads();
            if (e < np)
                transfer_chunk<kModeP2G, PLASTIC, VARIANT, THREADS, BS, false>(
                    TMPM_TRANSFER_ARGS, static_cast<int>(lists[e]), sp.step_index, sp.apply_force);
            else
                transfer_chunk<kModeG2P2G, PLASTIC, VARIANT, THREADS, BS, false>(
                    TMPM_TRANSFER_ARGS, static_cast<int>(lists[cap + (e - np)]), sp.step_index, sp.apply_force);
        }
    }
}

// A whole segment of a small scene (or batch) in one cooperative launch: table
// and pools cleared, the opening P2G, then `seg` substeps of grid update and
// fused transfer, the last one G2P-only, with a grid-wide barrier between
// phases; CTA c runs chunk c in every phase.
//
// At these sizes a substep's kernels are each a partial wave and the time goes
// into launches, the fork and join of the deferred chunks, the tails of
// dependent kernels and round trips to L2 for state the SM just wrote.  Here a
// phase starts one barrier after the last, the particle's state stays in
// registers and the chunk's record in shared memory, and only the grid goes
// through L2.  All chunks take the general path (128 registers a thread at two
// CTAs of 256 particles an SM), so nothing is deferred.  A frame of
// 8 substeps of 512 particles: 171 -> 139 us with the state and record kept and
// the clears inside (a substep 29,300 -> 22,900 cycles); of 16 substeps of 54,872
// particles 403 -> 341 us, 39,304 of snow 472 -> 399 us (kernel by kernel: 176,
// 483 and 613 us).
template <bool PLASTIC, int VARIANT, int THREADS, int BS>
__global__ void __launch_bounds__(THREADS, kSegmentThreads / THREADS) k_segment(TMPM_TRANSFER_PARAMS, int seg) {
    constexpr int TILE = segment_tile_nodes(THREADS);
    uint32_t *const arrived = cur.count + kBarrierWord;
    const size_t gtid = static_cast<size_t>(blockIdx.x) * THREADS + threadIdx.x;
    const size_t stride = static_cast<size_t>(gridDim.x) * THREADS;
    // CTAs above the chunk count only clear and update the grid
    const int chunk = blockIdx.x;
    const bool has_chunk = chunk * THREADS < n;
    {
        const size_t dirty = min(static_cast<size_t>(__ldcg(cur.count + kDirtyWord)), cur.pool_nodes);
        for (size_t t = gtid; t < dirty; t += stride) {
            cur.pool[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            next.pool[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (size_t t = gtid; t <= cur.mask; t += stride) {
            cur.keys[t] = kEmptyKey;
            cur.vals[t] = kPendingId;
        }
        if (gtid == 0) *cur.count = 0;
    }
    uint32_t target = gridDim.x;
    if (!grid_barrier(arrived, target, status)) return;
    ChunkState cs;
    if (has_chunk)
        transfer_chunk<kModeP2G, PLASTIC, VARIANT, THREADS, BS, false, TILE, true>(TMPM_TRANSFER_ARGS, chunk, -1, 0, &cs);
    GridTable a = next, b = cur;  // one table, two pools: `a` holds the nodes of the substep at hand
    for (int k = 0; k < seg; ++k) {
        if (!grid_barrier(arrived, target += gridDim.x, status)) return;
        if (!(*reinterpret_cast<volatile uint32_t *>(status) & kFatal))
            grid_nodes<VARIANT == kMulti, BS, has_obstacles(VARIANT)>(a, b.pool, sp, obstacles, planes, reactions, gtid,
                                                                      stride);
        if (!grid_barrier(arrived, target += gridDim.x, status)) return;
        const int force = k == 0 ? sp.apply_force : 0;
        if (has_chunk && k + 1 < seg)
            transfer_chunk<kModeG2P2G, PLASTIC, VARIANT, THREADS, BS, false, TILE, true>(
                P, n, classes, a, b, sp, obstacles, planes, reactions, status, cache, chunk, k, force, &cs);
        else if (has_chunk)
            transfer_chunk<kModeG2P, PLASTIC, VARIANT, THREADS, BS, false, TILE, true>(
                P, n, classes, a, b, sp, obstacles, planes, reactions, status, cache, chunk, k, force, &cs);
        float4 *const pool = a.pool;
        a.pool = b.pool;
        b.pool = pool;
    }
    if (gtid == 0) cur.count[kDirtyWord] = min(__ldcg(cur.count), cur.max_blocks) << (3 * BS);
    // the last CTA past every barrier leaves their words at zero
    if (threadIdx.x == 0 && atomicAdd(cur.count + kExitWord, 1u) == gridDim.x - 1) {
        *arrived = 0;
        cur.count[kExitWord] = 0;
    }
}
#undef TMPM_TRANSFER_ARGS
#undef TMPM_TRANSFER_PARAMS

}  // namespace

// Launch the transfer of `mode` for this variant; with `fj` the fused
// transfer runs in two tiers.
template <int V>
void launch_transfer_variant(int mode, const ParticleSoA &P, int n, const DevClass *classes, const GridTable &cur,
                             const GridTable &next, const SimParams &sp, const DevObstacle *obstacles,
                             const float *planes, double *reactions, uint32_t *status, int *cache,
                             cudaStream_t stream, const ForkJoin *fj) {
    // Plastic state exists for kPlainObst (with or without obstacles), kMulti
    // and kCpic; plastic and CPIC run the default shape and 4^3 blocks only.
    const bool pl = sp.has_plastic != 0;
    const int shape = (pl || V == kCpic) ? 0 : sp.shape;
    const bool big = !(pl || V == kCpic) && sp.block_shift == kBigBlockShift;
#define TMPM_ARGS P, n, classes, cur, next, sp, obstacles, planes, reactions, status, cache
    if constexpr (V != kCpic) {
        if (fj) {
            // The fused transfer as three kernels: the no-record chunks on
            // fj->side beside the fast kernel on `stream`, then (after both) the
            // chunks the fast kernel deferred.  The deferred kernels run one CTA
            // per SM over their lists; an empty list costs one short launch.
            const int sms = device_sm_count();
#define TMPM_FUSED(PL, T, B, BS) \
    do { \
        cudaEventRecord(fj->fork, stream); \
        cudaStreamWaitEvent(fj->side, fj->fork, 0); \
        k_transfer_deferred<true, PL, V, T, BS><<<sms, T, 0, fj->side>>>(TMPM_ARGS); \
        cudaEventRecord(fj->join, fj->side); \
        k_transfer_fast<PL, V, T, B, BS><<<dim3((n + (T) - 1) / (T)), T, 0, stream>>>(TMPM_ARGS); \
        cudaStreamWaitEvent(stream, fj->join, 0); \
        k_transfer_deferred<false, PL, V, T, BS><<<sms, T, 0, stream>>>(TMPM_ARGS); \
    } while (0)
#define TMPM_FUSED_SHAPES(BS) \
    do { \
        if (shape == 1) TMPM_FUSED(false, 128, 8, BS); \
        else if (shape == 2) TMPM_FUSED(false, 256, 3, BS); \
        else TMPM_FUSED(false, 256, TMPM_TRANSFER_MIN_BLOCKS, BS); \
    } while (0)
            if constexpr (V == kPlainObst) {
                if (pl) {
                    TMPM_FUSED(true, 256, TMPM_TRANSFER_MIN_BLOCKS, kBlockShift);
                    return;
                }
            }
            if (big) TMPM_FUSED_SHAPES(kBigBlockShift);
            else TMPM_FUSED_SHAPES(kBlockShift);
#undef TMPM_FUSED_SHAPES
#undef TMPM_FUSED
            return;
        }
    }
#define TMPM_LAUNCH(M, PL, T, B, BS) k_transfer<M, PL, V, T, B, BS><<<dim3((n + (T) - 1) / (T)), T, 0, stream>>>(TMPM_ARGS)
#define TMPM_LAUNCH_SHAPES(M, BS) \
    do { \
        if (shape == 1) TMPM_LAUNCH(M, false, 128, 8, BS); \
        else if (shape == 2) TMPM_LAUNCH(M, false, 256, 3, BS); \
        else TMPM_LAUNCH(M, false, 256, TMPM_TRANSFER_MIN_BLOCKS, BS); \
    } while (0)
#define TMPM_LAUNCH_MODE(M) \
    do { \
        if constexpr (V != kPlain) { \
            if (pl) { \
                TMPM_LAUNCH(M, true, 256, TMPM_TRANSFER_MIN_BLOCKS, kBlockShift); \
                return; \
            } \
        } \
        if constexpr (V == kCpic) TMPM_LAUNCH(M, false, 256, TMPM_TRANSFER_MIN_BLOCKS, kBlockShift); \
        else if (big) TMPM_LAUNCH_SHAPES(M, kBigBlockShift); \
        else TMPM_LAUNCH_SHAPES(M, kBlockShift); \
    } while (0)
    switch (mode) {
    case kModeP2G: TMPM_LAUNCH_MODE(kModeP2G); break;
    case kModeG2P2G: TMPM_LAUNCH_MODE(kModeG2P2G); break;
    default: TMPM_LAUNCH_MODE(kModeG2P); break;
    }
#undef TMPM_LAUNCH_MODE
#undef TMPM_LAUNCH_SHAPES
#undef TMPM_LAUNCH
#undef TMPM_ARGS
}

namespace {
// Launch k_segment if every chunk has a CTA resident at once and some are left for other streams.
template <bool PL, int V, int T, int BS>
bool try_segment(const ParticleSoA &P, int n, const DevClass *classes, const GridTable &cur, const GridTable &next,
                 const SimParams &sp, const DevObstacle *obstacles, const float *planes, double *reactions,
                 uint32_t *status, int *cache, int seg, cudaStream_t stream) {
    const int chunks = (n + T - 1) / T;
    const int smem = segment_tile_nodes(T) * static_cast<int>(sizeof(float4));
    int per_sm = 0;
    if (cudaFuncSetAttribute(k_segment<PL, V, T, BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_segment<PL, V, T, BS>, T, smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int room = whole_launch_room(per_sm * device_sm_count());
    if (chunks > room) return false;
    void *args[] = {const_cast<ParticleSoA *>(&P), &n, &classes, const_cast<GridTable *>(&cur),
                    const_cast<GridTable *>(&next), const_cast<SimParams *>(&sp), &obstacles, &planes, &reactions,
                    &status, &cache, &seg};
    if (cudaLaunchCooperativeKernel(k_segment<PL, V, T, BS>, dim3(std::min(room, std::max(chunks, kSegmentMinThreads / T))), dim3(T), args, smem, stream) ==
        cudaSuccess)
        return true;
    cudaGetLastError();
    return false;
}
}  // namespace

template <int V>
bool launch_segment_variant(const ParticleSoA &P, int n, const DevClass *classes, const GridTable &cur,
                            const GridTable &next, const SimParams &sp, const DevObstacle *obstacles,
                            const float *planes, double *reactions, uint32_t *status, int *cache, int seg,
                            cudaStream_t stream) {
#define TMPM_SEGMENT(PL, T, BS) \
    try_segment<PL, V, T, BS>(P, n, classes, cur, next, sp, obstacles, planes, reactions, status, cache, seg, stream)
    if (sp.has_plastic) {
        if constexpr (V == kPlainObst || V == kPlain) return TMPM_SEGMENT(true, 256, kBlockShift);
        return false;
    }
    const bool narrow = kLaunchShapes[sp.shape].threads == 128;
    if (sp.block_shift == kBigBlockShift)
        return narrow ? TMPM_SEGMENT(false, 128, kBigBlockShift) : TMPM_SEGMENT(false, 256, kBigBlockShift);
    return narrow ? TMPM_SEGMENT(false, 128, kBlockShift) : TMPM_SEGMENT(false, 256, kBlockShift);
#undef TMPM_SEGMENT
}

namespace {
template <int V, int T, int B, int BS>
void touch_shape() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_transfer_fast<false, V, T, B, BS>);
    cudaFuncGetAttributes(&a, k_transfer_deferred<true, false, V, T, BS>);
    cudaFuncGetAttributes(&a, k_transfer_deferred<false, false, V, T, BS>);
    cudaFuncGetAttributes(&a, k_transfer<kModeP2G, false, V, T, B, BS>);
    cudaFuncGetAttributes(&a, k_transfer<kModeG2P2G, false, V, T, B, BS>);
    cudaFuncGetAttributes(&a, k_transfer<kModeG2P, false, V, T, B, BS>);
    cudaFuncGetAttributes(&a, k_segment<false, V, T, BS>);
}
}  // namespace

// Load the kernels of every tuner candidate of this variant.
template <int V>
void preload_transfer_variant() {
    touch_shape<V, 256, TMPM_TRANSFER_MIN_BLOCKS, kBlockShift>();
    touch_shape<V, 128, 8, kBlockShift>();
    touch_shape<V, 256, 3, kBlockShift>();
    touch_shape<V, 256, TMPM_TRANSFER_MIN_BLOCKS, kBigBlockShift>();
    touch_shape<V, 128, 8, kBigBlockShift>();
    touch_shape<V, 256, 3, kBigBlockShift>();
}

#define TMPM_TRANSFER_VARIANT(V) \
    template void launch_transfer_variant<V>(int, const ParticleSoA &, int, const DevClass *, const GridTable &, \
                                                  const GridTable &, const SimParams &, const DevObstacle *, \
                                                  const float *, double *, uint32_t *, int *, cudaStream_t, \
                                                  const ForkJoin *);

#define TMPM_SEGMENT_VARIANT(V)                                                                                      \
    template bool launch_segment_variant<V>(const ParticleSoA &, int, const DevClass *, const GridTable &,           \
                                            const GridTable &, const SimParams &, const DevObstacle *, const float *, \
                                            double *, uint32_t *, int *, int, cudaStream_t);

}  // namespace tmpm
