// Device check of tmpm_tile.cuh's integer rules: the division-free split of padded
// tile indices (SplitP) at every stride and index that the tiles of the transfer
// kernels can have (the rollout's are between them), against integer division, and
// the fixed-point scale (pow2_scale, pow2_inverse) over its range of totals.
// Prints OK and exits 0, or the failures and exits 1.
#include <cstdio>

#include "../../tessera_b200/csrc/tmpm_transfer.cuh"

using namespace tmpm;

// Strides of a box of d1 x d2 (2 cells wider than its base cells, edges of at most
// 64) with at least three x planes in `entries`; one CTA per (d1, d2).
template <bool WIDE>
__global__ void check_split(int entries, unsigned *failures) {
    const int d1 = 3 + blockIdx.x, d2 = 3 + blockIdx.y;
    int s1, s2;
    tile_strides(d1, d2, s1, s2);
    if (3 * s1 > entries) return;
    const SplitP<WIDE> split(s1, s2);
    for (int t = threadIdx.x; t < entries; t += blockDim.x) {
        int x, y, z;
        split(t, x, y, z);
        const int r = t % s1;
        if (x != t / s1 || y != r / s2 || z != r % s2) atomicAdd(failures, 1u);
    }
}

// Largest power of two s with total * s <= 2^30, clamped to 2^-120 .. 2^120, and its inverse.
__global__ void check_scale(unsigned *failures) {
    const unsigned stride = gridDim.x * blockDim.x;
    // every total from 2^-100 to 2^100 in steps of 2^-9 of itself, and the floats beside the powers of two
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < 200u * 512u * 3u; k += stride) {
        const int bits = ((27 + static_cast<int>(k / (512u * 3u))) << 23) + (static_cast<int>(k / 3u % 512u) << 14) +
                         static_cast<int>(k % 3u) - 1;
        const float total = __int_as_float(bits), s = pow2_scale(total);
        const double product = static_cast<double>(fmaxf(total, 1e-30f)) * s;
        const int exponent = (__float_as_int(s) >> 23) - 127;
        const bool low = exponent == -120, high = exponent == 120;
        bool ok = (__float_as_int(s) & 0x7FFFFF) == 0 && s > 0.0f && pow2_inverse(s) == 1.0f / s;
        ok = ok && exponent >= -120 && exponent <= 120;
        ok = ok && (low || product <= 1073741824.0) && (high || 2.0 * product > 1073741824.0);
        if (!ok) atomicAdd(failures + 1, 1u);
    }
}

int main() {
    unsigned *failures = nullptr, host[4] = {};
    if (cudaMalloc(&failures, sizeof host) || cudaMemset(failures, 0, sizeof host)) return 3;
    const dim3 boxes(62, 62);  // d1, d2 in 3 .. 64
    check_split<false><<<boxes, 128>>>(tile_nodes(256), failures);
    check_split<true><<<boxes, 128>>>(segment_tile_nodes(256), failures + 2);
    check_scale<<<64, 256>>>(failures);
    if (cudaMemcpy(host, failures, sizeof host, cudaMemcpyDeviceToHost)) return 3;
    if (host[0] | host[1] | host[2]) {
        std::printf("split %u, wide split %u, scale %u\n", host[0], host[2], host[1]);
        return 1;
    }
    std::printf("OK\n");
    return 0;
}
