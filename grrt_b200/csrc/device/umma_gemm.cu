// BF16 GEMM on the sm_100a tensor cores for the learned surrogate:
//   C[M x N] = A[M x K] * B[N x K]^T   (A, B row-major BF16, i.e. K-major), or
//   C[M x N] = A[K x M]^T * B[K x N]   (A, B row-major BF16, i.e. MN-major, the
//   weight gradients: no transposed copies of the activations),
// FP32 accumulation in tensor memory, with a fused epilogue (bias, SiLU,
// SiLU-derivative gating, FP32/BF16 outputs, split-K partials).
//
// One CTA computes a 128-row tile and all N (<= 256) columns:
//   warp 0 lane 0: TMA producer (A and B K-blocks of 64 into a 4-stage ring,
//                  SWIZZLE_128B, completion on per-stage mbarriers);
//   warp 1 lane 0: MMA issuer (4 x tcgen05.mma K=16 per stage, commit frees
//                  the stage, a final commit signals the epilogue);
//   warps 0-7:     epilogue, each warp reads the 32 TMEM lanes (= tile rows) of
//                  its quadrant, warps 0-3 the even 16-column groups, 4-7 the odd.
// The epilogue is most of a tile: read by rows, stored by 64-byte row pieces.
// Every mbarrier wait is bounded; on timeout the CTA records an error code in
// *err, waits (bounded) for its TMA copies in flight, frees its tensor memory
// and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "launch_cache.h"
#include "sm100.cuh"
#include "umma_gemm.h"

namespace grrt_b200 {

namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kStages = 4;
constexpr uint32_t kBoxBytes = 64 * kBK * 2;  // an MN-major TMA box
constexpr int kThreads = 256;
constexpr int kPieceRow = 20;  // floats a row of an epilogue piece takes in shared memory
constexpr uint32_t kWaitLimit = 1u << 22;  // polls; a healthy wait needs a handful

struct GemmSmem {
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t done;
    uint32_t tmem_base;
    int failed;
};

__device__ __forceinline__ float silu(float z) { return sm100::silu_fast(z); }
__device__ __forceinline__ float silu_grad(float z) { return sm100::silu_grad_fast(z); }

// kMN: the operands are MN-major, a stage's tiles TMA boxes of 64 MN x kBK K.
template <bool kMN>
__global__ void __launch_bounds__(kThreads, 1)
umma_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const GemmEpilogue ep, int M, int N, int k_blocks_per_split, int k_blocks_total, int* err) {
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment for the swizzle atoms
    const uint32_t raw = sm100::smem_u32(smem_raw);
    unsigned char* tiles = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    const uint32_t a_bytes = kBM * kBK * 2, b_bytes = static_cast<uint32_t>(N) * kBK * 2;
    const uint32_t stage_bytes = a_bytes + b_bytes;
    GemmSmem* sh = reinterpret_cast<GemmSmem*>(tiles + kStages * stage_bytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM;
    const int split = blockIdx.y;
    const int kb0 = split * k_blocks_per_split;
    int kb1 = kb0 + k_blocks_per_split;
    if (kb1 > k_blocks_total) kb1 = k_blocks_total;
    const int nk = kb1 - kb0;
    // TMEM columns: a power of two >= 32 covering N
    uint32_t tcols = 32;
    while (tcols < static_cast<uint32_t>(N)) tcols <<= 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            sm100::mbar_init(&sh->full[s], 1);
            sm100::mbar_init(&sh->empty[s], 1);
        }
        sm100::mbar_init(&sh->done, 1);
        sh->failed = 0;
        sm100::fence_mbar_init();
        sm100::tma_prefetch_desc(&tmap_a);
        sm100::tma_prefetch_desc(&tmap_b);
    }
    if (warp == 0) {
        sm100::tmem_alloc(&sh->tmem_base, tcols);
        sm100::tmem_relinquish();
    }
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    const uint32_t idesc = sm100::idesc_bf16_f32(kBM, N, kMN);

    int issued = 0;  // producer: stages handed to TMA
    if (warp == 0 && lane == 0 && nk > 0) {
        for (int i = 0; i < nk; ++i) {
            const int s = i % kStages;
            if (i >= kStages && !sm100::mbar_wait(&sh->empty[s], ((i / kStages) - 1) & 1, kWaitLimit)) {
                atomicCAS(&sh->failed, 0, 1);
                break;
            }
            unsigned char* a_dst = tiles + s * stage_bytes;
            unsigned char* b_dst = a_dst + a_bytes;
            sm100::mbar_arrive_expect_tx(&sh->full[s], stage_bytes);
            const int kx = (kb0 + i) * kBK;
            if (kMN) {
                for (int j = 0; j < kBM / 64; ++j)
                    sm100::tma_load_2d(a_dst + j * kBoxBytes, &tmap_a, &sh->full[s], m0 + 64 * j, kx);
                for (int j = 0; j < N / 64; ++j)
                    sm100::tma_load_2d(b_dst + j * kBoxBytes, &tmap_b, &sh->full[s], 64 * j, kx);
            } else {
                sm100::tma_load_2d(a_dst, &tmap_a, &sh->full[s], kx, m0);
                sm100::tma_load_2d(b_dst, &tmap_b, &sh->full[s], kx, 0);
            }
            ++issued;
        }
    } else if (warp == 1 && lane == 0) {
        for (int i = 0; i < nk; ++i) {
            const int s = i % kStages;
            if (!sm100::mbar_wait(&sh->full[s], (i / kStages) & 1, kWaitLimit) ||
                *reinterpret_cast<volatile int*>(&sh->failed)) {
                atomicCAS(&sh->failed, 0, 2);
                break;
            }
            sm100::tc_fence_after();
            const uint32_t a_addr = sm100::smem_u32(tiles + s * stage_bytes);
            const uint32_t b_addr = a_addr + a_bytes;
            const uint64_t da = kMN ? sm100::desc_mnmajor_sw128(a_addr, kBoxBytes) : sm100::desc_kmajor_sw128(a_addr);
            const uint64_t db = kMN ? sm100::desc_mnmajor_sw128(b_addr, kBoxBytes) : sm100::desc_kmajor_sw128(b_addr);
            // 16 along K per step: 32 bytes of a K-major row, 16 rows of 128
            // bytes MN-major; the start-address field counts 16-byte units
            constexpr int kStep = kMN ? 16 * 128 / 16 : 2;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
                sm100::umma_f16(tmem, da + kStep * k, db + kStep * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
            sm100::umma_commit(&sh->empty[s]);
        }
        sm100::umma_commit(&sh->done);  // also completes when nothing was issued
    }
    __syncwarp();

    // epilogue: wait for the accumulator
    bool ok = sm100::mbar_wait(&sh->done, 0, kWaitLimit);
    if (!ok) atomicCAS(&sh->failed, 0, 3);
    sm100::tc_fence_after();
    __syncthreads();
    const bool good = (*reinterpret_cast<volatile int*>(&sh->failed) == 0);
    const int quad = warp & 3;  // the TMEM lanes a warp may read
    if (good) {
        // Every stage has been consumed (the commit on `done` follows all MMAs), so
        // each warp turns its 32 x 16 pieces round in its part of the ring: a
        // lane reads a row of the accumulator, but 4 lanes store 64 consecutive
        // bytes of a row (padded rows of 20 floats: no bank conflicts).
        float* const piece = reinterpret_cast<float*>(tiles) + warp * (32 * kPieceRow);
        const uint32_t t_row = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        const size_t zoff = ep.split_stride * static_cast<size_t>(split);
        const bool wide = ((reinterpret_cast<uintptr_t>(ep.gate_z) | (static_cast<size_t>(ep.ld_gate) * 4)) & 15) == 0;
        const int sub = lane >> 2, col4 = (lane & 3) * 4;  // of the row groups of 8: row and columns this lane moves
        const int row0 = m0 + quad * 32 + sub;
        for (int c0 = 16 * (warp >> 2); c0 < N; c0 += 32) {
            float4 z[4], bias = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (ep.gate_z) {  // in flight while the accumulator is read
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const int r = row0 + 8 * g;
                    if (r >= M) continue;
                    const float* zp = ep.gate_z + static_cast<size_t>(r) * ep.ld_gate + c0 + col4;
                    z[g] = wide ? *reinterpret_cast<const float4*>(zp) : make_float4(zp[0], zp[1], zp[2], zp[3]);
                }
            }
            if (ep.bias) {
                const float* bp = ep.bias + c0 + col4;
                bias = make_float4(bp[0], bp[1], bp[2], bp[3]);
            }
            float v[16];
            __syncwarp();  // the load is of the whole warp; rows past M were skipped lane by lane above
            sm100::tmem_ld16(t_row + static_cast<uint32_t>(c0), v);
            if (nk <= 0) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<float4*>(piece + lane * kPieceRow + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            __syncwarp();
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int r = row0 + 8 * g;
                if (r >= M) continue;
                float4 x = *reinterpret_cast<const float4*>(piece + (sub + 8 * g) * kPieceRow + col4);
                if (ep.bias) {
                    x.x += bias.x;
                    x.y += bias.y;
                    x.z += bias.z;
                    x.w += bias.w;
                }
                if (ep.gate_z) {  // backward through SiLU: x *= silu'(z)
                    x.x *= silu_grad(z[g].x);
                    x.y *= silu_grad(z[g].y);
                    x.z *= silu_grad(z[g].z);
                    x.w *= silu_grad(z[g].w);
                }
                if (ep.out_f32)
                    *reinterpret_cast<float4*>(ep.out_f32 + zoff + static_cast<size_t>(r) * ep.ld_f32 + c0 + col4) = x;
                if (ep.out_bf16) {
                    if (ep.act == kActSilu) x = make_float4(silu(x.x), silu(x.y), silu(x.z), silu(x.w));
                    alignas(8) const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(x.x, x.y),
                                                            __floats2bfloat162_rn(x.z, x.w)};
                    *reinterpret_cast<uint2*>(ep.out_bf16 + static_cast<size_t>(r) * ep.ld_bf16 + c0 + col4) =
                        *reinterpret_cast<const uint2*>(h);
                }
            }
            __syncwarp();  // the piece is free again
        }
    }
    if (!good && threadIdx.x == 0) {
        atomicExch(err, sh->failed);
    }
    // a failed producer may still have copies in flight: wait for them (bounded)
    if (!good && warp == 0 && lane == 0) {
        for (int i = 0; i < issued; ++i) sm100::mbar_wait(&sh->full[i % kStages], (i / kStages) & 1, kWaitLimit);
    }
    sm100::tc_fence_before();
    __syncthreads();
    if (warp == 0) sm100::tmem_dealloc(tmem, tcols);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Row-major BF16 matrix [rows x cols] with row pitch ld (elements), box
// [box_rows x 64], SWIZZLE_128B; out-of-range elements read as zero.
bool make_tmap(CUtensorMap* m, const void* base, int rows, int cols, int ld, int box_rows) {
    auto fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

size_t umma_gemm_smem_bytes(int N) {
    return 1024 + static_cast<size_t>(kStages) * (kBM * kBK * 2 + static_cast<size_t>(N) * kBK * 2) + sizeof(GemmSmem);
}

namespace {

// Outputs of a GEMM: 16-byte accesses (the gate is read in any alignment).
bool epilogue_ok(const GemmEpilogue& ep, int splits) {
    if (ep.out_bf16 && ((ep.ld_bf16 % 8) != 0 || (reinterpret_cast<uintptr_t>(ep.out_bf16) & 15))) return false;
    if (ep.out_f32 && ((ep.ld_f32 % 4) != 0 || (reinterpret_cast<uintptr_t>(ep.out_f32) & 15))) return false;
    // split-K writes raw FP32 partials only
    return splits == 1 || !(ep.out_bf16 || ep.bias || ep.gate_z || !ep.out_f32 || ep.split_stride == 0);
}

template <bool kMN>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, int splits,
                   const GemmEpilogue& ep, int* d_err, cudaStream_t stream) {
    const int kbt = K / kBK;
    const int per = (kbt + splits - 1) / splits;
    splits = (kbt + per - 1) / per;  // every split gets at least one K-block
    const size_t smem = umma_gemm_smem_bytes(N);
    // the shared-memory attribute is set once per device, with that device current
    struct Attr {
        cudaError_t err = cudaSuccess;
    };
    const Attr& attr = per_device_shape<Attr>([](int) {
        Attr a;
        a.err = cudaFuncSetAttribute(umma_gemm_kernel<kMN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(umma_gemm_smem_bytes(256)));
        return a;
    });
    if (attr.err != cudaSuccess) return attr.err;
    dim3 grid((M + kBM - 1) / kBM, splits);
    umma_gemm_kernel<kMN><<<grid, kThreads, smem, stream>>>(ta, tb, ep, M, N, per, kbt, d_err);
    return cudaGetLastError();
}

}  // namespace

cudaError_t umma_gemm_bf16(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K,
                           int splits, const GemmEpilogue& ep, int* d_err, cudaStream_t stream) {
    // shapes the kernel supports; everything else is a caller error
    if (M <= 0 || N < 16 || N > 256 || (N % 16) != 0 || K <= 0 || (K % kBK) != 0 || splits < 1) return cudaErrorInvalidValue;
    if ((lda % 8) != 0 || (ldb % 8) != 0 || lda < K || ldb < K) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return cudaErrorInvalidValue;
    if (!epilogue_ok(ep, splits)) return cudaErrorInvalidValue;
    CUtensorMap ta, tb;
    if (!make_tmap(&ta, A, M, K, lda, kBM) || !make_tmap(&tb, B, N, K, ldb, N)) return cudaErrorInvalidValue;
    return launch<false>(ta, tb, M, N, K, splits, ep, d_err, stream);
}

cudaError_t umma_gemm_tn_bf16(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K,
                              int splits, const GemmEpilogue& ep, int* d_err, cudaStream_t stream) {
    if (M <= 0 || N < 64 || N > 256 || (N % 64) != 0 || K <= 0 || (K % kBK) != 0 || splits < 1) return cudaErrorInvalidValue;
    if ((lda % 8) != 0 || (ldb % 8) != 0 || lda < M || ldb < N) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return cudaErrorInvalidValue;
    if (!epilogue_ok(ep, splits)) return cudaErrorInvalidValue;
    CUtensorMap ta, tb;  // boxes of 64 columns x kBK rows; columns past M read as zero
    if (!make_tmap(&ta, A, K, M, lda, kBK) || !make_tmap(&tb, B, K, N, ldb, kBK)) return cudaErrorInvalidValue;
    return launch<true>(ta, tb, M, N, K, splits, ep, d_err, stream);
}

}  // namespace grrt_b200
