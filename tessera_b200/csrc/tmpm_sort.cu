// tmpm_sort.cu -- stable LSD radix sort of (u32 key, u32 value) pairs.
//
// Used to bring particles into block order (Morton key of their 4^3 block).
// Above kSmallSort keys each 8-bit pass is three kernels:
//   k_hist    per-tile digit histogram (tile = 4096 keys), digit-major layout
//   k_scan    per-digit exclusive scan over tiles + digit totals
//   k_scatter stable scatter: each warp ranks 32 keys at a time with
//             __match_any_sync, so equal digits keep their input order.
// Up to kSmallSort keys the whole sort is four kernels (k_small_keys,
// 3 x k_small_pass).

#include <algorithm>

#include "tmpm_device.cuh"

namespace tmpm {

namespace {

constexpr int kSortThreads = 256;
constexpr int kItemsPerThread = 16;
constexpr int kTile = kSortThreads * kItemsPerThread;  // 4096
constexpr int kWarps = kSortThreads / 32;
constexpr int kWarpItems = kTile / kWarps;  // 512 contiguous keys per warp

__global__ void __launch_bounds__(kSortThreads) k_hist(const uint32_t *__restrict__ keys, int n, int shift,
                                                       uint32_t *hist, int tiles) {
    __shared__ uint32_t counts[256];
    counts[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kTile;
#pragma unroll 4
    for (int j = 0; j < kItemsPerThread; ++j) {
        int idx = base + j * kSortThreads + threadIdx.x;
        if (idx < n) atomicAdd(&counts[(keys[idx] >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    hist[static_cast<size_t>(threadIdx.x) * tiles + blockIdx.x] = counts[threadIdx.x];
}

// One CTA per digit: exclusive scan of hist[d][0..tiles) in place; totals[d] = sum.
__global__ void __launch_bounds__(kSortThreads) k_scan(uint32_t *hist, int tiles, uint32_t *totals) {
    __shared__ uint32_t warp_sums[kWarps];
    __shared__ uint32_t carry;
    uint32_t *row = hist + static_cast<size_t>(blockIdx.x) * tiles;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int start = 0; start < tiles; start += kSortThreads) {
        int idx = start + threadIdx.x;
        uint32_t v = idx < tiles ? row[idx] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        uint32_t warp_prefix = 0, chunk_total = 0;
        for (int w = 0; w < kWarps; ++w) {
            if (w < warp) warp_prefix += warp_sums[w];
            chunk_total += warp_sums[w];
        }
        uint32_t c = carry;
        if (idx < tiles) row[idx] = c + warp_prefix + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry = c + chunk_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(kSortThreads) k_scatter(const uint32_t *__restrict__ keys_in,
                                                          const uint32_t *__restrict__ vals_in, uint32_t *keys_out,
                                                          uint32_t *vals_out, int n, int shift,
                                                          const uint32_t *__restrict__ hist, int tiles,
                                                          const uint32_t *__restrict__ totals) {
    __shared__ uint32_t digit_base[256];
    __shared__ uint32_t wcount[kWarps][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // exclusive scan of the 256 digit totals (each CTA redoes this small scan)
    {
        uint32_t v = totals[threadIdx.x];
        uint32_t incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        __shared__ uint32_t sums[kWarps];
        if (lane == 31) sums[warp] = incl;
        __syncthreads();
        uint32_t pre = 0;
        for (int w = 0; w < warp; ++w) pre += sums[w];
        digit_base[threadIdx.x] = pre + incl - v + hist[static_cast<size_t>(threadIdx.x) * tiles + blockIdx.x];
        for (int w = 0; w < kWarps; ++w) wcount[w][threadIdx.x] = 0;
    }
    __syncthreads();

    const int base = blockIdx.x * kTile + warp * kWarpItems;
    const unsigned lt_mask = (1u << lane) - 1u;
    uint32_t k_reg[kItemsPerThread], v_reg[kItemsPerThread], r_reg[kItemsPerThread];
#pragma unroll
    for (int r = 0; r < kItemsPerThread; ++r) {
        int idx = base + r * 32 + lane;
        bool ok = idx < n;
        uint32_t key = ok ? keys_in[idx] : 0u;
        uint32_t digit = ok ? ((key >> shift) & 0xFFu) : 256u;
        unsigned peers = __match_any_sync(0xffffffffu, digit);
        uint32_t before = 0;
        if (ok) before = wcount[warp][digit];
        __syncwarp();
        int leader = __ffs(peers) - 1;
        if (ok && lane == leader) wcount[warp][digit] = before + __popc(peers);
        __syncwarp();
        k_reg[r] = key;
        v_reg[r] = ok ? vals_in[idx] : 0u;
        r_reg[r] = before + __popc(peers & lt_mask);
    }
    __syncthreads();
    // exclusive scan over warps, per digit
    {
        uint32_t run = 0;
        for (int w = 0; w < kWarps; ++w) {
            uint32_t c = wcount[w][threadIdx.x];
            wcount[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItemsPerThread; ++r) {
        int idx = base + r * 32 + lane;
        if (idx >= n) continue;
        uint32_t digit = (k_reg[r] >> shift) & 0xFFu;
        uint32_t pos = digit_base[digit] + wcount[warp][digit] + r_reg[r];
        keys_out[pos] = k_reg[r];
        vals_out[pos] = v_reg[r];
    }
}


// ------------------------------------------------------------- small sorts
//
// A sort of some 10^5 keys is bound by launches and by kernels that fill a
// fraction of the GPU, not by its ~2 MB of traffic.  So: smaller tiles (2048
// keys: 98 CTAs at 200,000 keys, not 49), 9 or 10 bits a pass (three passes
// instead of four for 27- and 30-bit keys), and one kernel per pass.  A pass
// needs the digit histogram of every tile of its input; the kernel before it
// counts them while it writes that input (the key kernel its own tile's, a pass
// with global atomics on the tile each key lands in), and every CTA of the pass
// sums the columns it needs itself (tiles x 2 KB from L2), which replaces the
// scan kernel.  With 128 tiles or fewer that sum stays at a few microseconds; it
// grows with the square of the count, so larger sorts keep the scan.
// Measured at 200,003 keys (one call of the allocation-free binning): 106 us before, 49 us now; the
// pass kernels run 98 CTAs of 512 threads.
constexpr int kSmallThreads = 512;
constexpr int kSmallItems = 4;
constexpr int kSmallTile = kSmallThreads * kSmallItems;  // 2048
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallWarpItems = kSmallTile / kSmallWarps;  // 128 contiguous keys per warp

// Keys of a tile, their digit histogram for the first pass, and zeroes for the
// histograms of the later passes (`hist`: three [tiles][2^BITS] arrays).
template <int BITS>
__global__ void __launch_bounds__(kSmallThreads) k_small_keys(BinSource src, uint32_t *keys, uint32_t *hist, int tiles) {
    constexpr int kDigits = 1 << BITS;
    __shared__ uint32_t counts[kDigits];
    const size_t later = static_cast<size_t>(tiles) * kDigits;
    uint32_t *const row = hist + static_cast<size_t>(blockIdx.x) * kDigits;
    for (int d = threadIdx.x; d < kDigits; d += kSmallThreads) {
        counts[d] = 0;
        row[later + d] = 0;
        row[2 * later + d] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallItems; ++j) {
        const int i = blockIdx.x * kSmallTile + j * kSmallThreads + threadIdx.x;
        if (i >= src.n) break;
        const uint32_t key = bin_key(src, i);
        keys[i] = key;
        atomicAdd(&counts[key & (kDigits - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSmallThreads) row[d] = counts[d];
}

// One pass over digit (key >> shift): PASS 0 takes the identity as values; the
// last pass (2) counts nothing for a next one.
template <int BITS, int PASS>
__global__ void __launch_bounds__(kSmallThreads) k_small_pass(const uint32_t *__restrict__ keys_in,
                                                              const uint32_t *__restrict__ vals_in, uint32_t *keys_out,
                                                              uint32_t *vals_out, int n, uint32_t *hist, int tiles) {
    constexpr int kDigits = 1 << BITS, kPer = kDigits / kSmallThreads, kShift = BITS * PASS;
    constexpr uint32_t kMask = kDigits - 1;
    __shared__ uint32_t base[kDigits];
    __shared__ uint16_t wcount[kSmallWarps][kDigits];
    __shared__ uint32_t sums[kSmallWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t later = static_cast<size_t>(tiles) * kDigits;
    const uint32_t *const mine = hist + PASS * later;

    // this thread's keys, loaded beside the histogram sums
    const int first = blockIdx.x * kSmallTile + warp * kSmallWarpItems + lane;
    uint32_t key[kSmallItems], val[kSmallItems];
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int idx = first + 32 * r;
        key[r] = idx < n ? keys_in[idx] : 0u;
        val[r] = PASS == 0 ? static_cast<uint32_t>(idx) : (idx < n ? vals_in[idx] : 0u);
    }
    for (int d = threadIdx.x; d < kSmallWarps * kDigits / 2; d += kSmallThreads)
        reinterpret_cast<uint32_t *>(&wcount[0][0])[d] = 0;
    // per digit: keys in earlier tiles, keys in all; thread t owns digits t * kPer ..
    uint32_t before[kPer], total[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) before[p] = total[p] = 0;
#pragma unroll 8
    for (int t = 0; t < tiles; ++t)
#pragma unroll
        for (int p = 0; p < kPer; ++p) {
            const uint32_t c = mine[static_cast<size_t>(t) * kDigits + threadIdx.x * kPer + p];
            if (t < static_cast<int>(blockIdx.x)) before[p] += c;
            total[p] += c;
        }
    uint32_t own = 0;
#pragma unroll
    for (int p = 0; p < kPer; ++p) own += total[p];
    uint32_t incl = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    uint32_t run = incl - own;
    for (int w = 0; w < warp; ++w) run += sums[w];
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
        base[threadIdx.x * kPer + p] = run + before[p];
        run += total[p];
    }
    // rank within the warp's 128 keys, in order
    const unsigned lt_mask = (1u << lane) - 1u;
    uint32_t rank[kSmallItems];
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const bool ok = first + 32 * r < n;
        const uint32_t digit = ok ? (key[r] >> kShift) & kMask : kDigits;
        const unsigned peers = __match_any_sync(0xffffffffu, digit);
        uint32_t seen = 0;
        if (ok) seen = wcount[warp][digit];
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) wcount[warp][digit] = static_cast<uint16_t>(seen + __popc(peers));
        __syncwarp();
        rank[r] = seen + __popc(peers & lt_mask);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSmallThreads) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kSmallWarps; ++w) {
            const uint32_t c = wcount[w][d];
            wcount[w][d] = static_cast<uint16_t>(sum);
            sum += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        if (first + 32 * r >= n) continue;
        const uint32_t digit = (key[r] >> kShift) & kMask;
        const uint32_t pos = base[digit] + wcount[warp][digit] + rank[r];
        if (keys_out) keys_out[pos] = key[r];
        vals_out[pos] = val[r];
        if (PASS < 2)
            atomicAdd(hist + (PASS + 1) * later + static_cast<size_t>(pos / kSmallTile) * kDigits +
                          ((key[r] >> (kShift + BITS)) & kMask),
                      1u);
    }
}

template <int BITS>
void small_sort(const BinSource &src, SortBuffers &sb, uint32_t *keys_out, uint32_t *vals_out, cudaStream_t stream) {
    const int tiles = (src.n + kSmallTile - 1) / kSmallTile;
    k_small_keys<BITS><<<tiles, kSmallThreads, 0, stream>>>(src, sb.keys[0], sb.hist, tiles);
    k_small_pass<BITS, 0><<<tiles, kSmallThreads, 0, stream>>>(sb.keys[0], nullptr, sb.keys[1], sb.vals[1], src.n,
                                                               sb.hist, tiles);
    k_small_pass<BITS, 1><<<tiles, kSmallThreads, 0, stream>>>(sb.keys[1], sb.vals[1], sb.keys[0], sb.vals[0], src.n,
                                                               sb.hist, tiles);
    k_small_pass<BITS, 2><<<tiles, kSmallThreads, 0, stream>>>(sb.keys[0], sb.vals[0], keys_out, vals_out, src.n,
                                                               sb.hist, tiles);
}

}  // namespace

size_t sort_hist_words(size_t cap) {
    const size_t large = 256 * ((cap + kTile - 1) / kTile);
    const size_t small = 3 * ((std::min(cap, kSmallSort) + kSmallTile - 1) / kSmallTile) * 1024;
    return std::max(large, small);
}

int bin_and_sort(const BinSource &src, SortBuffers &sb, int bits, uint32_t *keys_out, uint32_t *vals_out,
                 cudaStream_t stream) {
    const bool out = vals_out != nullptr;
    if (static_cast<size_t>(src.n) <= kSmallSort && bits <= 30) {
        if (!out) {
            keys_out = sb.keys[1];
            vals_out = sb.vals[1];
        }
        if (bits <= 27) small_sort<9>(src, sb, keys_out, vals_out, stream);
        else small_sort<10>(src, sb, keys_out, vals_out, stream);
        return 1;
    }
    launch_bin_keys(src, nullptr, sb.keys[0], sb.vals[0], stream);
    const int r = radix_sort_pairs(sb, src.n, bits, stream);
    if (out) {
        cudaMemcpyAsync(vals_out, sb.vals[r], sizeof(uint32_t) * src.n, cudaMemcpyDeviceToDevice, stream);
        if (keys_out)
            cudaMemcpyAsync(keys_out, sb.keys[r], sizeof(uint32_t) * src.n, cudaMemcpyDeviceToDevice, stream);
    }
    return r;
}

int radix_sort_pairs(SortBuffers &sb, int n, int bits, cudaStream_t stream) {
    if (n <= 0) return 0;
    const int tiles = (n + kTile - 1) / kTile;
    int cur = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        k_hist<<<tiles, kSortThreads, 0, stream>>>(sb.keys[cur], n, shift, sb.hist, tiles);
        k_scan<<<256, kSortThreads, 0, stream>>>(sb.hist, tiles, sb.totals);
        k_scatter<<<tiles, kSortThreads, 0, stream>>>(sb.keys[cur], sb.vals[cur], sb.keys[cur ^ 1], sb.vals[cur ^ 1], n,
                                                      shift, sb.hist, tiles, sb.totals);
        cur ^= 1;
    }
    return cur;
}

}  // namespace tmpm
