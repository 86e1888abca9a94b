// tmpm_kernels.cu -- the MLS-MPM substep on sm_100a: the grid update, binning,
// row and readback kernels, and the dispatch of the transfer kernels.
//
// One substep n of the resident path is two kernels:
//   k_grid(n):      v = p / m + g dt, walls, obstacles, reactions
//                   (world.rs:401-417, gpu.wgsl:772-819 / 1056-1108)
//   k_transfer(n):  G2P of step n fused with P2G of step n+1
//                   (world.rs:419-464 then 378-399; gpu.wgsl:821-1019, 711-770)
// A batch opens with a P2G-only transfer and closes with a G2P-only transfer,
// which alone writes velocity and the affine matrix back to HBM.  The transfer
// kernels are in tmpm_transfer.cuh.

#include "tmpm_grid.cuh"

namespace tmpm {

namespace {

// Grid update (grid_nodes) as a kernel of its own.
template <bool MULTI, int BS, bool OBST>
__global__ void __launch_bounds__(256) k_grid(GridTable g, GridTable nxt, SimParams sp,
                                               const DevObstacle *__restrict__ obstacles,
                                               const float *__restrict__ planes, double *reactions, uint32_t *status) {
    __shared__ int s_abort;
    // empty the deferred-chunk lists that the next transfer (step_index) fills
    if (sp.defer && blockIdx.x == 0 && threadIdx.x == 0) {
        sp.defer[0] = 0;
        sp.defer[1] = 0;
        sp.defer[2 + ((sp.step_index + 1) & 1)] = 0;
    }
    if (threadIdx.x == 0) s_abort = (*reinterpret_cast<volatile uint32_t *>(status) & kFatal) != 0;
    __syncthreads();
    if (s_abort) return;
    grid_nodes<MULTI, BS, OBST>(g, nxt.pool, sp, obstacles, planes, reactions,
                                static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x,
                                static_cast<size_t>(gridDim.x) * blockDim.x);
}

__global__ void k_clear_table(GridTable g) {
    const size_t gtid = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t s = gtid; s <= g.mask; s += stride) {
        g.keys[s] = kEmptyKey;
        g.vals[s] = kPendingId;
    }
    if (gtid == 0) {
        g.count[0] = 0;
        g.count[kDirtyWord] = ~0u;
    }
}

__global__ void k_bin_keys(BinSource src, int32_t *cells, uint32_t *keys, uint32_t *vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= src.n) return;
    keys[i] = bin_key(src, i, cells);
    if (vals) vals[i] = static_cast<uint32_t>(i);
}

// dst[j] = src[perm[s(j)]] for every particle field.  With `interleave` = T,
// each full chunk of T sorted particles (one transfer CTA) is stored
// transposed: thread kk of the chunk (warp w = kk / 32, lane l = kk % 32) holds
// sorted particle l * G + w with G = T / 32, so the 32 lanes of
// a warp take one particle from each of 32 consecutive groups of G
// (cell-sorted: one or two cells each) and their stencils do not collide on
// the same shared-memory node.  The last, partial chunk is stored in sorted
// order.
__global__ void k_gather(ParticleSoA src, ParticleSoA dst, const uint32_t *__restrict__ perm, int n, int interleave) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    int sj = j;
    if (interleave) {  // interleave = particles per transfer CTA (0: stored in sorted order)
        const int chunk = j / interleave;
        if ((chunk + 1) * interleave <= n) {
            const int kk = j - chunk * interleave;
            sj = chunk * interleave + lane_cell(kk % 32) * (interleave / 32) + kk / 32;
        }
    }
    int s = static_cast<int>(perm[sj]);
    const size_t cs = src.cap, cd = dst.cap;
    for (int c = 0; c < 3; ++c) {
        dst.x[c * cd + j] = src.x[c * cs + s];
        dst.v[c * cd + j] = src.v[c * cs + s];
        dst.pl[c * cd + j] = src.pl[c * cs + s];
    }
    for (int c = 0; c < 9; ++c) {
        dst.C[c * cd + j] = src.C[c * cs + s];
        dst.F[c * cd + j] = src.F[c * cs + s];
    }
    dst.cls[j] = src.cls[s];
    dst.widx[j] = src.widx[s];
}

// Device rows back in world order: out[c * stride + widx[j]] = row c of stored
// particle j, for the 27 f32 components (x, v, C, F, plastic), so the host
// applies a readback sequentially instead of scattering through the sort
// permutation.
__global__ void k_unsort(ParticleSoA P, int n, float *__restrict__ out, size_t stride, uint32_t *nonfinite) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const size_t cap = P.cap, w = P.widx[j];
    bool finite = true;
    for (int c = 0; c < 3; ++c) {
        const float x = P.x[c * cap + j], v = P.v[c * cap + j], p = P.pl[c * cap + j];
        finite = finite && isfinite(x) && isfinite(v) && isfinite(p);
        out[c * stride + w] = x;
        out[(3 + c) * stride + w] = v;
        out[(24 + c) * stride + w] = p;
    }
    for (int c = 0; c < 9; ++c) {
        const float a = P.C[c * cap + j], f = P.F[c * cap + j];
        finite = finite && isfinite(a) && isfinite(f);
        out[(6 + c) * stride + w] = a;
        out[(15 + c) * stride + w] = f;
    }
    if (nonfinite && !finite) atomicOr(nonfinite, 1u);
}

template <int BS>
__global__ void k_dump_grid(GridTable g, int32_t *cells, float4 *values, uint32_t *count, uint32_t capacity) {
    uint32_t nblocks = min(*g.count, g.max_blocks);
    constexpr int kM = (1 << BS) - 1;
    size_t nodes = static_cast<size_t>(nblocks) << (3 * BS);
    for (size_t node = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; node < nodes;
         node += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float4 mp = g.pool[node];
        if (mp.x == 0.0f) continue;
        uint32_t slot = atomicAdd(count, 1u);
        if (slot >= capacity) continue;
        int4 c = g.coords[node >> (3 * BS)];
        int l = static_cast<int>(node) & ((1 << (3 * BS)) - 1);
        cells[3 * slot] = (c.x << BS) + (l >> (2 * BS));
        cells[3 * slot + 1] = (c.y << BS) + ((l >> BS) & kM);
        cells[3 * slot + 2] = (c.z << BS) + (l & kM);
        values[slot] = mp;
    }
}

__global__ void k_snapshot(ParticleSoA P, int n, const DevClass *__restrict__ classes, float4 *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t cap = P.cap;
    const DevClass &k = classes[P.cls[i] & kClassMask];
    uint32_t w = P.widx[i];
    out[2 * w] = make_float4(P.x[i], P.x[cap + i], P.x[2 * cap + i], k.mass);
    out[2 * w + 1] = make_float4(P.v[i], P.v[cap + i], P.v[2 * cap + i], k.volume);
}

}  // namespace

int device_sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

void launch_transfer(int mode, const ParticleSoA &P, int n, const DevClass *classes, const GridTable &cur,
                     const GridTable &next, const SimParams &sp, const DevObstacle *obstacles, const float *planes,
                     double *reactions, uint32_t *status, int *cache, cudaStream_t stream, const ForkJoin *fj) {
    if (n <= 0) return;
    // the two tiers run the fused transfer only, and not for CPIC or a batch with plastic state
    if (mode != kModeG2P2G || !sp.defer || sp.cpic || (sp.multi && sp.has_plastic)) fj = nullptr;
#define TMPM_VARIANT(V) \
    launch_transfer_variant<V>(mode, P, n, classes, cur, next, sp, obstacles, planes, reactions, status, cache, stream, fj)
    // plastic state and CPIC run with the obstacle contact compiled in, with or without obstacles
    if (sp.multi) TMPM_VARIANT(kMulti);
    else if (sp.cpic) TMPM_VARIANT(kCpic);
    else if (sp.has_plastic || sp.num_obstacles > 0) TMPM_VARIANT(kPlainObst);
    else TMPM_VARIANT(kPlain);
#undef TMPM_VARIANT
}

bool launch_small_segment(const ParticleSoA &P, int n, const DevClass *classes, const GridTable &cur,
                          const GridTable &next, const SimParams &sp, const DevObstacle *obstacles,
                          const float *planes, double *reactions, uint32_t *status, int *cache, int seg,
                          cudaStream_t stream) {
    if (n <= 0 || seg <= 0 || sp.cpic) return false;
    SimParams one = sp;
    one.defer = nullptr;  // nothing is deferred: every chunk runs the general path
#define TMPM_VARIANT(V)                                                                                            \
    launch_segment_variant<V>(P, n, classes, cur, next, one, obstacles, planes, reactions, status, cache, seg, stream)
    if (sp.multi) return TMPM_VARIANT(kMulti);
    // plastic state without obstacles: the contact's out-of-line call takes
    // registers the return map needs (864 -> 336 bytes of stack)
    if (sp.num_obstacles > 0) return TMPM_VARIANT(kPlainObst);
    return TMPM_VARIANT(kPlain);
#undef TMPM_VARIANT
}

void launch_grid_update(const GridTable &g, const GridTable &next, const SimParams &sp, const DevObstacle *obstacles,
                        const float *planes, double *reactions, uint32_t *status, cudaStream_t stream) {
    int blocks = device_sm_count() * 8;
    const bool obst = !sp.multi && sp.num_obstacles > 0;
#define TMPM_GRID(MU, BS, OB) k_grid<MU, BS, OB><<<blocks, 256, 0, stream>>>(g, next, sp, obstacles, planes, reactions, status)
    if (sp.block_shift == kBigBlockShift) {
        if (sp.multi) TMPM_GRID(true, kBigBlockShift, false);
        else if (obst) TMPM_GRID(false, kBigBlockShift, true);
        else TMPM_GRID(false, kBigBlockShift, false);
    } else {
        if (sp.multi) TMPM_GRID(true, kBlockShift, false);
        else if (obst) TMPM_GRID(false, kBlockShift, true);
        else TMPM_GRID(false, kBlockShift, false);
    }
#undef TMPM_GRID
}

void preload_launch_shapes(bool multi, bool obstacles) {
    if (multi) preload_transfer_variant<kMulti>();
    else if (obstacles) preload_transfer_variant<kPlainObst>();
    else preload_transfer_variant<kPlain>();
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, multi ? k_grid<true, kBlockShift, false>
                                    : (obstacles ? k_grid<false, kBlockShift, true> : k_grid<false, kBlockShift, false>));
    cudaFuncGetAttributes(&a, multi ? k_grid<true, kBigBlockShift, false>
                                    : (obstacles ? k_grid<false, kBigBlockShift, true>
                                                 : k_grid<false, kBigBlockShift, false>));
    cudaGetLastError();
}

void launch_clear_table(const GridTable &g, const GridTable &other, int block_shift, cudaStream_t stream) {
    int blocks = device_sm_count() * 4;
    k_clear_table<<<blocks, 256, 0, stream>>>(g);
    // new block ids start from zero again: both pools start zero-filled
    const size_t bytes = (static_cast<size_t>(g.max_blocks) << (3 * block_shift)) * sizeof(float4);
    cudaMemsetAsync(g.pool, 0, bytes, stream);
    if (other.pool != g.pool) cudaMemsetAsync(other.pool, 0, bytes, stream);
}

void launch_bin_keys(const BinSource &src, int32_t *cells, uint32_t *keys, uint32_t *vals, cudaStream_t stream) {
    if (src.n <= 0) return;
    k_bin_keys<<<(src.n + 255) / 256, 256, 0, stream>>>(src, cells, keys, vals);
}

void launch_resort(ParticleSoA &src, ParticleSoA &dst, int n, int keep, const DevClass *classes, const SimParams &sp,
                   SortBuffers &sb, cudaStream_t stream) {
    if (n <= 0) return;
    const BinSource bins{src.x, src.cap, n, sp.s0.inv_h, src.cls, classes, sp.multi ? sp.scenes : nullptr};
    const int r = bin_and_sort(bins, sb, sp.multi ? kSortBitsBatch : kSortBitsScene, nullptr, nullptr, stream);
    const int interleave = sp.multi ? 0 : kLaunchShapes[sp.shape].threads;
    if (keep > 0) k_gather<<<(keep + 255) / 256, 256, 0, stream>>>(src, dst, sb.vals[r], keep, interleave);
}

void launch_dump_grid(const GridTable &g, int32_t *cells, float4 *values, uint32_t *count, uint32_t capacity,
                      int block_shift, cudaStream_t stream) {
    if (block_shift == kBigBlockShift)
        k_dump_grid<kBigBlockShift><<<device_sm_count() * 4, 256, 0, stream>>>(g, cells, values, count, capacity);
    else
        k_dump_grid<kBlockShift><<<device_sm_count() * 4, 256, 0, stream>>>(g, cells, values, count, capacity);
}

void launch_unsort(const ParticleSoA &P, int n, float *out, size_t stride, cudaStream_t stream, uint32_t *nonfinite) {
    if (n <= 0) return;
    k_unsort<<<(n + 255) / 256, 256, 0, stream>>>(P, n, out, stride, nonfinite);
}

void launch_snapshot(const ParticleSoA &P, int n, const DevClass *classes, float4 *out, cudaStream_t stream) {
    if (n <= 0) return;
    k_snapshot<<<(n + 255) / 256, 256, 0, stream>>>(P, n, classes, out);
}

}  // namespace tmpm
