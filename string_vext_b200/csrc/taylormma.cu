// The matrix product of taylormma.cuh on the fifth-generation tensor cores.
//
// 4,096 rows x 28,800 regions x 448 sums (60^3 x 64 layered field, forward +
// adjoint): 0.44 ms, 317 GFLOP in three TF32 products, against 2.06 ms as packed
// FP32 FMA (taylor_eval_kernel's tiles) that two thirds of the FMA pipe bounded.
// Bound by the tensor pipe, 73 % of its cycles active (44^3), then by the
// operands' way from L2: 96 KB a chunk of 32 sums against about 1,600 cycles of
// products.  128 x 256 tiles with both accumulators in TMEM are the largest that
// leave two stages of 96 KB in shared memory.
//
// Error: the parts hold 22-23 bits and the sums are ordered by falling degree,
// so that the accumulator stays far below the value until the last few products.
// Against the 64-bit product of the FP32 sums with the exact matrix, its rms error is
// 0.27-0.37 of that of 435 FP32 FMAs in sequence, its largest 0.12-0.31 (layered 60^3
// x 64, skewed 47^3 x 50 and 60^3 x 64, four smaller ones; energies 2.8e-9-2.0e-8 K,
// gradients 7.8e-9-4.2e-8 K/A rms).  The matrix split from FP64 would give 0.25-0.35,
// with the product of the low parts too 0.23-0.32.
#include "taylormma.cuh"

namespace vext {

constexpr uint32_t kPartA = kMmaM * kMmaK * 4, kPartB = kMmaN * kMmaK * 4;   // bytes
constexpr uint32_t kStageMma = 2 * (kPartA + kPartB);
constexpr int kMmaStages = 2;
constexpr uint32_t kMmaThreads = 192;
constexpr uint32_t kMmaSmem = 1024 + kMmaStages * kStageMma + 128;
constexpr uint32_t kTmemColumns = 2 * kMmaN;   // two accumulators

struct MmaArgs {
    const float *a, *b;
    int row_tiles, tiles;      // tiles = row tiles x region tiles
    int n_regions, out_len;
    float *out;
    int *status;
};

// Shared-memory descriptor of a K-major operand part with the 128-byte swizzle:
// start / 16, groups of eight rows 1024 bytes apart, version 1, layout 2.
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    // FP32 accumulator, TF32 operands, both K-major, N / 8, M / 16
    constexpr uint32_t idesc =
        (1u << 4) | (2u << 7) | (2u << 10) | ((kMmaN / 8) << 17) | ((kMmaM / 16) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
          "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

#define TCGEN05_BEFORE() asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory")
#define TCGEN05_AFTER() asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory")

// One CTA per SM takes every gridDim-th tile.  Warp 0 brings the operands
// (two bulk copies a chunk of 32 sums), warp 1 issues the products, warps 2-5
// read a finished accumulator while the other one fills.
__global__ void __launch_bounds__(kMmaThreads, 1) taylor_mma_kernel(MmaArgs a) {
    extern __shared__ unsigned char raw[];
    unsigned char *smem = raw + (1024 - (smem_addr(raw) & 1023)) % 1024;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kMmaStages * kStageMma);
    uint64_t *full = bar, *empty = bar + 2, *acc_full = bar + 4, *acc_empty = bar + 6;
    uint32_t *tmem_word = reinterpret_cast<uint32_t *>(bar + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
            mbar_init(acc_full + s, 1);
            mbar_init(acc_empty + s, 4);
        }
        fence_mbar_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(tmem_word)),
                     "r"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    TCGEN05_BEFORE();
    __syncthreads();
    TCGEN05_AFTER();
    const uint32_t tmem = *tmem_word;
    if (warp == 0) {
        if (lane == 0) {
            unsigned it = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < a.tiles; t += gridDim.x) {
                const float *ga = a.a + (size_t)(t % a.row_tiles) * kMmaChunks * (2 * kPartA / 4);
                const float *gb = a.b + (size_t)(t / a.row_tiles) * kMmaChunks * (2 * kPartB / 4);
                for (int c = 0; c < kMmaChunks; ++c, ++it) {
                    const int s = it & 1;
                    ok = mbar_wait_bounded(empty + s, ((it >> 1) & 1) ^ 1, a.status);
                    if (!ok) break;
                    unsigned char *st = smem + s * kStageMma;
                    mbar_arrive_expect_tx(full + s, kStageMma);
                    bulk_g2s(st, ga + (size_t)c * (2 * kPartA / 4), 2 * kPartA, full + s);
                    bulk_g2s(st + 2 * kPartA, gb + (size_t)c * (2 * kPartB / 4), 2 * kPartB,
                             full + s);
                }
            }
            // own copies end before the CTA does, also after a wait that gave up
            for (unsigned k = it > 2 ? it - 2 : 0; k < it; ++k)
                mbar_drain(full + (k & 1), (k >> 1) & 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            unsigned it = 0, j = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < a.tiles; t += gridDim.x, ++j) {
                const uint32_t d = tmem + (j & 1) * kMmaN;
                ok = mbar_wait_bounded(acc_empty + (j & 1), ((j >> 1) & 1) ^ 1, a.status);
                if (!ok) break;
                TCGEN05_AFTER();
                for (int c = 0; c < kMmaChunks; ++c, ++it) {
                    const int s = it & 1;
                    ok = mbar_wait_bounded(full + s, (it >> 1) & 1, a.status);
                    if (!ok) break;
                    TCGEN05_AFTER();
                    const uint32_t sa = smem_addr(smem + s * kStageMma), sb = sa + 2 * kPartA;
                    const uint64_t ah = mma_desc(sa), al = mma_desc(sa + kPartA),
                                   bh = mma_desc(sb), bl = mma_desc(sb + kPartB);
                    // eight sums (32 bytes) an instruction; small products first
#pragma unroll
                    for (int k = 0; k < kMmaK / 8; ++k) mma_tf32(d, al + 2 * k, bh + 2 * k, c + k);
#pragma unroll
                    for (int k = 0; k < kMmaK / 8; ++k) mma_tf32(d, ah + 2 * k, bl + 2 * k, 1);
#pragma unroll
                    for (int k = 0; k < kMmaK / 8; ++k) mma_tf32(d, ah + 2 * k, bh + 2 * k, 1);
                    mma_commit(empty + s);
                }
                if (ok) mma_commit(acc_full + (j & 1));
            }
            // products in flight end before the shared memory goes
            for (unsigned k = it > 2 ? it - 2 : 0; k < it; ++k)
                mbar_drain(empty + (k & 1), (k >> 1) & 1);
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3;   // the TMEM lanes this warp can read
        unsigned j = 0;
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++j) {
            const bool ok = mbar_wait_bounded(acc_full + (j & 1), (j >> 1) & 1, a.status);
            if (!__all_sync(0xffffffffu, ok)) break;
            TCGEN05_AFTER();
            const int row = t % a.row_tiles * kMmaM + quarter * 32 + lane;
            const int region0 = t / a.row_tiles * kMmaN;
            const uint32_t d = tmem + (j & 1) * kMmaN + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < kMmaN; c += 32) {
                if (region0 + c >= a.n_regions) break;
                uint32_t v[32];
                tmem_load32(d + c, v);
                float *out = a.out + (size_t)(region0 + c) * a.out_len + row;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (region0 + c + i < a.n_regions && row < a.out_len)
                        out[(size_t)i * a.out_len] = __uint_as_float(v[i]);
            }
            TCGEN05_BEFORE();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                                 smem_addr(acc_empty + (j & 1)))
                             : "memory");
        }
    }
    TCGEN05_BEFORE();
    __syncthreads();
    TCGEN05_AFTER();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemColumns));
}

size_t taylor_workspace_sites(const RegionSet &rs) {
    const size_t tiles = ((size_t)rs.n_regions + kMmaN - 1) / kMmaN;
    return tiles * kMmaN * kTaylorPad * 2;
}

int taylor_mma(const float *matrix, int row_tiles, const float *sums, int n_regions, int out_len,
               float *out, int *status, cudaStream_t stream) {
    MmaArgs a;
    a.a = matrix;
    a.b = sums;
    a.row_tiles = row_tiles;
    a.tiles = row_tiles * ((n_regions + kMmaN - 1) / kMmaN);
    a.n_regions = n_regions;
    a.out_len = out_len;
    a.out = out;
    a.status = status;
    int dev = 0, sms = 0;
    VEXT_CUDA(cudaGetDevice(&dev));
    VEXT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    VEXT_CUDA(cudaFuncSetAttribute(taylor_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kMmaSmem));
    taylor_mma_kernel<<<std::min(sms, a.tiles), kMmaThreads, kMmaSmem, stream>>>(a);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace vext
