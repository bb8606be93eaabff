// BF16 GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA) for the move-ordering
// MLP.  No reference counterpart: the reference has no learned component.
//
//   C[M x N] (fp32 accumulate in TMEM) = A[M x K] * B[N x K]^T
//
// Either operand may be stored the other way round in memory (A as [K x M], B as [K x N], rows
// contiguous): the tensor core reads such a tile MN-major, so a backward product needs no
// transposed copy.  One CTA computes one 128 x BN tile over a span of K:
//   warp 0 lane 0  TMA producer: 2-D tiled copies (128-byte swizzle) into a ring of stages;
//   warp 1 lane 0  MMA issuer: four tcgen05.mma.kind::f16 (M=128, N=BN, K=16) per stage,
//                  tcgen05.commit frees the stage, a final commit signals the epilogue;
//   warps 0-3      epilogue: tcgen05.ld 32 columns at a time from their TMEM lane quadrant,
//                  bias, ReLU or the backward ReLU mask, then rows of 128 bytes staged in the
//                  (by then idle) ring with the swizzle and stored by TMA, 4 KB per store.
// K is accumulated in one order whatever BN is, so results do not depend on the tile choice.
// Every mbarrier wait is bounded by a 2 s deadline; on expiry the kernel records an error,
// skips the remaining tensor-core work and still frees its TMEM.
//
// Bound: the output's stores for the logits (K = 256: 84 MB of fp32 per 4,096 rows), latency
// of the K loop for the narrow layers.  Against a thread-per-row epilogue with scalar stores
// and one 128 x 256 tile per SM (one B200, device time, 4,096 rows): logits 253 -> 31 us, hidden
// layers 61 (K = 1,088) and 56 (K = 256) -> 9 and 5 us, gradient of the last hidden layer
// 68 -> 31 us (bound by the operand copies, about 32 B per cycle and SM), weight gradients
// 45 to 51 -> 7 to 21 us without the transposed copies (45 us for the logits' gradient alone).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "mlp.h"

namespace tdp {
namespace mlp {
namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
// The ring takes 96 KB for either tile width, so two CTAs share an SM and one's epilogue
// overlaps the other's loads.  (64-wide tiles with one CTA per SM and a ring of 192 KB: the same
// time where one wave covers the tiles, up to twice as long where it does not.)
__host__ __device__ constexpr int ring_stages(int bn) { return bn == 64 ? 4 : 3; }
__host__ __device__ constexpr int ring_bytes(int bn) { return ring_stages(bn) * (A_BYTES + bn * BK * 2); }
__host__ __device__ constexpr int smem_bytes(int bn) { return ring_bytes(bn) + bn * 4 + 1024 + 256; }
constexpr unsigned long long kWaitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bounded wait for the completion of the phase with the given parity.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *err) {
    const unsigned long long start = now_ns();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (now_ns() - start > kWaitNs) {
            atomicExch(err, 1);
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(src)
                 : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle.  K-major: a row of 64 K values is 128
// bytes, 8-row groups 1024 B apart.  MN-major: 64 M (or N) values of one K are 128 bytes, 8-K
// groups 1024 B apart, the next 64 M (or N) values one 64 x 64 box (8192 B) on.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, bool mnMajor) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);                          // start address
    d |= (uint64_t)(mnMajor ? (8192u >> 4) : 1u) << 16;              // leading byte offset (unused K-major)
    d |= (uint64_t)(1024u >> 4) << 32;                               // stride byte offset
    d |= (uint64_t)1u << 46;                                         // descriptor version (sm_100)
    d |= (uint64_t)2u << 61;                                         // SWIZZLE_128B
    return d;
}

// Instruction descriptor: kind::f16, A/B bf16, D fp32, M=128, N=BN; bits 15 and 16: A, B MN-major.
__host__ __device__ constexpr uint32_t instr_desc(int bn, bool mnA, bool mnB) {
    return (1u << 4)              // D format f32
           | (1u << 7)            // A format bf16
           | (1u << 10)           // B format bf16
           | ((mnA ? 1u : 0u) << 15) | ((mnB ? 1u : 0u) << 16)
           | ((uint32_t)(bn >> 3) << 17)
           | ((uint32_t)(BM >> 4) << 24);
}

enum Output { kOutBf16, kOutF32, kOutScalar };  // TMA stores, or element stores to any address

template <int BN, bool MN_A, bool MN_B, Output OUT>
__global__ void __launch_bounds__(128, 2)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
    constexpr int STAGES = ring_stages(BN), B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float *biasTile = reinterpret_cast<float *>(smem + STAGES * STAGE_BYTES);
    uint64_t *full = reinterpret_cast<uint64_t *>(biasTile + BN);
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;
    uint32_t *tmemSlot = reinterpret_cast<uint32_t *>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tileN = blockIdx.x, tileM = blockIdx.y;
    const int allTiles = (p.K + BK - 1) / BK;
    const int k0 = blockIdx.z * p.tilesPerSplit, kTiles = min(p.tilesPerSplit, allTiles - k0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(full + s), 1);
            mbar_init(smem_u32(empty + s), 1);
        }
        mbar_init(smem_u32(done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmemSlot)),
                     "r"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int c = threadIdx.x; c < BN; c += 128)
        biasTile[c] = p.bias && tileN * BN + c < p.N ? p.bias[tileN * BN + c] : 0.f;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmemSlot;

    if (warp == 0 && lane == 0) {
        for (int kt = 0; kt < kTiles; ++kt) {
            const int s = kt % STAGES, round = kt / STAGES;
            // a timed-out wait has set p.error; the later waits give up the same way
            if (round > 0 && !mbar_wait(smem_u32(empty + s), (uint32_t)((round - 1) & 1), p.error)) break;
            const uint32_t a = smem_u32(smem + s * STAGE_BYTES);
            const uint32_t b = a + A_BYTES;
            const uint32_t bar = smem_u32(full + s);
            const int k = (k0 + kt) * BK;
            mbar_expect_tx(bar, STAGE_BYTES);
            if (MN_A) {
#pragma unroll
                for (int i = 0; i < BM / 64; ++i) tma_load_2d(a + i * 8192, &tmA, tileM * BM + i * 64, k, bar);
            } else {
                tma_load_2d(a, &tmA, k, tileM * BM, bar);
            }
            if (MN_B) {
#pragma unroll
                for (int i = 0; i < BN / 64; ++i) tma_load_2d(b + i * 8192, &tmB, tileN * BN + i * 64, k, bar);
            } else {
                tma_load_2d(b, &tmB, k, tileN * BN, bar);
            }
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = instr_desc(BN, MN_A, MN_B);
        bool ok = true;
        for (int kt = 0; kt < kTiles && ok; ++kt) {
            const int s = kt % STAGES, round = kt / STAGES;
            if (!mbar_wait(smem_u32(full + s), (uint32_t)(round & 1), p.error)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(smem + s * STAGE_BYTES);
            const uint32_t b = a + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
                // 16 K values on: 32 bytes along a K-major row, two 8-K groups MN-major
                const uint64_t da = smem_desc(a + kk * (MN_A ? 2048 : 32), MN_A);
                const uint64_t db = smem_desc(b + kk * (MN_B ? 2048 : 32), MN_B);
                const uint32_t accumulate = (kt > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(empty + s))
                         : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(done))
                     : "memory");
    }
    __syncwarp();

    // Epilogue: every thread owns one row (TMEM lane) of the tile.  After `done` every MMA has
    // read its operands, so the ring is free for staging.
    const bool ready = mbar_wait(smem_u32(done), 0u, p.error);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int row = tileM * BM + warp * 32 + lane;
    if (ready) {
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
            uint32_t r[32];
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                  "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                  "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (p.bias || p.relu) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    float v = __uint_as_float(r[j]);
                    if (p.bias) v += biasTile[c0 + j];
                    if (p.relu) v = fmaxf(v, 0.0f);
                    r[j] = __float_as_uint(v);
                }
            }
            if (OUT == kOutScalar) {
                if (row < p.M) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int col = tileN * BN + c0 + j;
                        if (col < p.N) {
                            const size_t o = (size_t)row * (size_t)p.ldo + (size_t)col;
                            if (p.outF32) p.outF32[o] = __uint_as_float(r[j]);
                            if (p.outBf16) p.outBf16[o] = __float2bfloat16_rn(__uint_as_float(r[j]));
                        }
                    }
                }
            } else if (OUT == kOutF32) {
                // 32 columns are a 128-byte row: 16-byte chunk q of row `lane` at q ^ (lane & 7)
                uint8_t *const stage = smem + (warp * (BN / 32) + c0 / 32) * 4096;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    *reinterpret_cast<uint4 *>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                        make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0 && tileN * BN + c0 < p.N && tileM * BM + warp * 32 < p.M) {
                    tma_store_2d(&tmC, smem_u32(stage), tileN * BN + c0, (int)blockIdx.z * p.M + tileM * BM + warp * 32);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else {
                // 64 bf16 columns are a 128-byte row: this half of it
                uint8_t *const stage = smem + (warp * (BN / 64) + c0 / 64) * 4096;
                uint32_t packed[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
                    packed[j] = *reinterpret_cast<const uint32_t *>(&v);
                }
                if (p.mask && row < p.M) {
                    // backward ReLU: the gradient is zero where the activation is not positive
                    const uint4 *act = reinterpret_cast<const uint4 *>(p.mask + (size_t)row * p.N + tileN * BN + c0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 v = tileN * BN + c0 + 8 * q < p.N ? __ldg(act + q) : make_uint4(0u, 0u, 0u, 0u);
                        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const __nv_bfloat162 a2 = *reinterpret_cast<const __nv_bfloat162 *>(&w[j]);
                            const uint32_t low = __low2float(a2) <= 0.f ? 0u : 0xFFFFu;
                            const uint32_t high = __high2float(a2) <= 0.f ? 0u : 0xFFFF0000u;
                            packed[4 * q + j] &= low | high;
                        }
                    }
                }
                const int half = (c0 & 32) ? 4 : 0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<uint4 *>(stage + lane * 128 + (((q + half) ^ (lane & 7)) << 4)) =
                        make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
                if (half) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && tileN * BN + c0 - 32 < p.N && tileM * BM + warp * 32 < p.M) {
                        tma_store_2d(&tmC, smem_u32(stage), tileN * BN + c0 - 32, tileM * BM + warp * 32);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            }
        }
        // the staged rows leave before the CTA does
        if (OUT != kOutScalar && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
    }
}

// ---------------------------------------------------------------- tensor maps
using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn(std::string &err) {
    static std::mutex mu;
    static EncodeFn fn = nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !ptr) {
            err = "cuTensorMapEncodeTiled is not available";
            return nullptr;
        }
        fn = reinterpret_cast<EncodeFn>(ptr);
    }
    return fn;
}

// rows x cols row-major with `stride` elements per row, box = boxRows x 128 bytes, 128B swizzle.
bool make_map(CUtensorMap *map, const void *base, int rows, int cols, int stride, int boxRows, bool f32,
              std::string &err) {
    EncodeFn fn = encode_fn(err);
    if (!fn) return false;
    const int size = f32 ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0 || (stride * size) % 16 != 0) {
        err = "gemm operand must be 16-byte aligned with a row length that is a multiple of 8";
        return false;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)stride * size};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / size), (cuuint32_t)boxRows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                          const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        err = "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
        return false;
    }
    return true;
}

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const GemmParams);

// The kernels that exist: forward products in both tile widths and all outputs, gradients of
// the input (B stored [K x N]) and of the weights (both operands stored [K x .]).
constexpr int kForms = 8;
const Kernel kKernels[kForms] = {
    gemm_bf16_kernel<64, false, false, kOutBf16>,   gemm_bf16_kernel<64, false, false, kOutF32>,
    gemm_bf16_kernel<64, false, false, kOutScalar>, gemm_bf16_kernel<128, false, false, kOutBf16>,
    gemm_bf16_kernel<128, false, false, kOutF32>,   gemm_bf16_kernel<128, false, false, kOutScalar>,
    gemm_bf16_kernel<64, false, true, kOutBf16>,    gemm_bf16_kernel<128, true, true, kOutF32>,
};
constexpr int kFormInputGrad = 6, kFormWeightGrad = 7;

int launch(int form, int bn, int splits, CUtensorMap &ma, CUtensorMap &mb, CUtensorMap &mc, const GemmParams &p,
           cudaStream_t stream, std::string &err) {
    const dim3 grid((p.N + bn - 1) / bn, (p.M + BM - 1) / BM, splits);
    kKernels[form]<<<grid, 128, smem_bytes(bn), stream>>>(ma, mb, mc, p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("gemm launch: ") + cudaGetErrorString(e);
        return -3;
    }
    return 0;
}

}  // namespace

int prepare(std::string &err) {
    // a kernel's shared-memory limit is raised on each device by itself
    static std::mutex mu;
    static std::vector<bool> raised;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (e == cudaSuccess && (size_t)device >= raised.size()) raised.resize((size_t)device + 1, false);
        if (e == cudaSuccess && !raised[(size_t)device]) {
            for (int f = 0; f < kForms && e == cudaSuccess; ++f)
                e = cudaFuncSetAttribute(kKernels[f], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         std::max(smem_bytes(64), smem_bytes(128)));
            raised[(size_t)device] = e == cudaSuccess;
        }
    }
    if (e != cudaSuccess) {
        cudaGetLastError();  // reported here, not by the next launch's check
        err = std::string("gemm set-up: ") + cudaGetErrorString(e);
        return -3;
    }
    return encode_fn(err) ? 0 : -1;
}

int gemm_bf16(const void *A, const void *B, int M, int N, int K, const float *bias, int relu, void *out, int outFp32,
              int ldo, int *errorFlag, cudaStream_t stream, std::string &err) {
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !out || !errorFlag) {
        err = "gemm: bad arguments";
        return -1;
    }
    GemmParams p{};
    p.M = M;
    p.N = N;
    p.K = K;
    p.tilesPerSplit = (K + BK - 1) / BK;
    p.bias = bias;
    p.relu = relu;
    p.outBf16 = outFp32 ? nullptr : static_cast<__nv_bfloat16 *>(out);
    p.outF32 = outFp32 ? static_cast<float *>(out) : nullptr;
    p.ldo = ldo > 0 ? ldo : N;
    p.error = errorFlag;
    // 64-wide tiles while one wave of two CTAs per SM holds them all (148 SMs), else 128-wide ones,
    // which read A half as often.  Device time 64- / 128-wide: 4,096 x 256 x 1,088 8.9 / 9.3 us,
    // 8,192 x 256 x 1,088 (256 narrow tiles) 10.0 / 10.4, 512 x 5,120 x 256 (320) 8.8 / 7.0,
    // 4,096 x 5,120 x 256 41 / 30.
    const long long narrow = (long long)((N + 63) / 64) * ((M + BM - 1) / BM);
    const int bn = narrow <= 2 * 148 ? 64 : 128;
    CUtensorMap ma, mb, mc;
    std::memset(&mc, 0, sizeof(mc));
    if (!make_map(&ma, A, M, K, K, BM, false, err) || !make_map(&mb, B, N, K, K, bn, false, err)) return -1;
    if (prepare(err) != 0) return -3;
    // TMA stores where the output allows them (16-byte base and row stride)
    const size_t size = outFp32 ? 4 : 2;
    const bool tma = (reinterpret_cast<uintptr_t>(out) & 15u) == 0 && ((size_t)p.ldo * size) % 16 == 0 && p.ldo >= N;
    if (tma && !make_map(&mc, out, M, N, p.ldo, 32, outFp32 != 0, err)) return -3;
    return launch((bn == 128 ? 3 : 0) + (!tma ? 2 : outFp32 ? 1 : 0), bn, 1, ma, mb, mc, p, stream, err);
}

int gemm_input_grad(const __nv_bfloat16 *grad, const __nv_bfloat16 *W, int rows, int outDim, int inDim,
                    const __nv_bfloat16 *act, __nv_bfloat16 *out, int *errorFlag, cudaStream_t stream,
                    std::string &err) {
    GemmParams p{};
    p.M = rows;
    p.N = inDim;
    p.K = outDim;
    p.tilesPerSplit = (outDim + BK - 1) / BK;
    p.mask = act;
    p.ldo = inDim;
    p.error = errorFlag;
    CUtensorMap ma, mb, mc;
    if (!make_map(&ma, grad, rows, outDim, outDim, BM, false, err) ||
        !make_map(&mb, W, outDim, inDim, inDim, BK, false, err) ||
        !make_map(&mc, out, rows, inDim, inDim, 32, false, err))
        return -1;
    if (prepare(err) != 0) return -3;
    return launch(kFormInputGrad, 64, 1, ma, mb, mc, p, stream, err);
}

// K spans for about one CTA per SM, each of at least four K tiles (the partial sums are read again
// by the optimiser, so more spans cost there what they gain here).
int weight_grad_splits(int rows, int outDim, int inDim) {
    const int tiles = ((outDim + BM - 1) / BM) * ((inDim + 127) / 128);
    const int kTiles = (rows + BK - 1) / BK;
    const int wanted = std::max(1, std::min(kTiles / 4, (148 + tiles / 2) / tiles));
    const int per = (kTiles + wanted - 1) / wanted;
    return (kTiles + per - 1) / per;
}

int gemm_weight_grad(const __nv_bfloat16 *grad, const __nv_bfloat16 *act, int rows, int outDim, int inDim,
                     float *partials, int *errorFlag, cudaStream_t stream, std::string &err) {
    if (outDim % BM != 0) {
        err = "gemm: weight gradient rows must be a multiple of 128";
        return -1;
    }
    const int splits = weight_grad_splits(rows, outDim, inDim);
    GemmParams p{};
    p.M = outDim;
    p.N = inDim;
    p.K = rows;
    p.tilesPerSplit = ((rows + BK - 1) / BK + splits - 1) / splits;
    p.ldo = inDim;
    p.error = errorFlag;
    CUtensorMap ma, mb, mc;
    if (!make_map(&ma, grad, rows, outDim, outDim, BK, false, err) ||
        !make_map(&mb, act, rows, inDim, inDim, BK, false, err) ||
        !make_map(&mc, partials, splits * outDim, inDim, inDim, 32, true, err))
        return -1;
    if (prepare(err) != 0) return -3;
    return launch(kFormWeightGrad, 128, splits, ma, mb, mc, p, stream, err);
}

}  // namespace mlp
}  // namespace tdp
