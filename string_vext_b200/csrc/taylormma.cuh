// The expansions' values at single sites as a matrix product on the tensor
// cores (taylormma.cu): [rows of sites x sums] . [sums x regions], both factors
// split into two TF32 parts each (x = hi + lo to 2^-23), three products.
//
// Both operands are stored in global memory as the shared-memory images the
// instruction reads: tiles of T rows x 32 sums, K-major with the 128-byte
// swizzle, for each (row tile, 32 sums) the hi and then the lo part.
#pragma once

#include "taylor.cuh"

namespace vext {

constexpr int kMmaM = 128, kMmaN = 256, kMmaK = 32;   // rows of sites, regions, sums of a tile
constexpr int kMmaChunks = kTaylorPad / kMmaK;
static_assert(kTaylorPad % kMmaK == 0, "whole chunks");

// Place of each sum along K: falling degree, after the padding, so that the
// running sums stay small until the last, largest terms.
struct MmaOrder {
    unsigned short at[kTaylorSums];
};
__host__ __device__ constexpr MmaOrder mma_order() {
    MmaOrder o{};
    int next = kTaylorPad - kTaylorSums;
    for (int degree = kTaylorOrder; degree >= kTaylorLow; --degree)
        for (int r = 0; r < kTaylorRoles; ++r) {
            int base = role_start(r);
            for (int c = 0; c < 3; ++c) {
                const int m = role_column(r, c);
                if (m < 0) continue;
                int at = base;
                for (int l = m; l <= kTaylorOrder; ++l)
                    for (int k = 0; l + 2 * k <= kTaylorOrder; ++k) {
                        if (l + 2 * k < kTaylorLow) continue;
                        for (int cs = 0; cs < (m ? 2 : 1); ++cs, ++at)
                            if (l + 2 * k == degree) o.at[at] = (unsigned short)next++;
                    }
                base = at;
            }
        }
    return o;
}
static __device__ const MmaOrder kMmaOrder = mma_order();

// x into row `row`, sum `k` of an operand in tiles of T rows.
template <int T>
__device__ __forceinline__ void mma_store_split(float *operand, int row, int k, float x) {
    uint32_t hb, lb;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(x));
    const float hi = __uint_as_float(hb & 0xffffe000u);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lb) : "f"(x - hi));
    const int r = row % T, kk = k % kMmaK;
    float *p = operand + ((size_t)(row / T) * kMmaChunks + k / kMmaK) * 2 * T * kMmaK +
               r * kMmaK + (((kk >> 2) ^ (r & 7)) << 2) + (kk & 3);
    p[0] = hi;
    p[T * kMmaK] = __uint_as_float(lb & 0xffffe000u);
}

// out[region][row] for row < out_len (<= kMmaM x row_tiles).
int taylor_mma(const float *matrix, int row_tiles, const float *sums, int n_regions, int out_len,
               float *out, int *status, cudaStream_t stream);

}  // namespace vext
