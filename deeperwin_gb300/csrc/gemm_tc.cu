// Persistent tcgen05 tensor-core GEMM for sm_103a.
//
//   C[M, N] = epilogue( A[M, K] @ W[N, K]^T )
//
// * A and W are BF16 (NP = 1) or split-BF16 (NP = 2: x = hi + lo, three MMAs per K step:
//   A_hi W_hi + A_hi W_lo + A_lo W_hi, all accumulated in FP32 in TMEM).
// * Warp roles (320 threads): warp 0 = TMA producer, warp 1 = MMA issuer (one elected lane),
//   warps 2-9 = epilogue (warp w drains TMEM lanes 32 (w % 4) .. +31; the two warps of a lane
//   quarter take alternate 32-column chunks).
// * Shared-memory ring of S stages (128-byte swizzled K-major tiles), two TMEM accumulators
//   so the epilogue of tile i overlaps the main loop of tile i + 1, one CTA per SM looping
//   over output tiles.
// * Epilogue: value-channel bias, per-(walker, channel) row bias and tanh on value rows (the tangent
//   passes' layers are in gemm_jet.cu). Results are written to swizzled shared-memory staging tiles (two per warp, so the staging
//   of one chunk overlaps the TMA store of the previous one) and stored with TMA.
// Every mbarrier wait is bounded; on timeout the kernel records an error flag, stops
// issuing, waits (bounded) for its TMA loads in flight, frees its TMEM and returns.
#include "gemm_tc.cuh"
#include <stdlib.h>
#include <string.h>
#include <algorithm>

namespace dw {

__device__ int g_tc_error = 0;

// ------------------------------------------------------------------ tensor maps
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

}  // namespace

// 2-D tensor map: dims {cols (inner), rows}, row stride ld elements, box {box_cols, box_rows},
// swizzle of box_cols * element size bytes (128 or 64).
int make_map(CUtensorMap* map, const void* base, int64_t rows, int cols, int64_t ld, int box_cols, int box_rows,
             bool f32) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return DW_ERR_UNSUPPORTED;
    const int es = f32 ? 4 : 2;
    const int span = box_cols * es;
    if (((uintptr_t)base & 15) || (ld * es) % 16 || (span != 128 && span != 64)) return DW_ERR_ARG;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * es};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                    const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? DW_OK : DW_ERR_ARG;
}

// 3-D tensor map {cols (inner), rows, walkers}: row stride ld and walker stride wstride elements,
// box {box_cols, box_rows, box_w}, swizzle of box_cols * element size bytes (128 or 64).
int make_map3(CUtensorMap* map, const void* base, int64_t nw, int rows, int cols, int64_t ld, int64_t wstride,
              int box_cols, int box_rows, int box_w, bool f32) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return DW_ERR_UNSUPPORTED;
    const int es = f32 ? 4 : 2;
    const int span = box_cols * es;
    if (((uintptr_t)base & 15) || (ld * es) % 16 || (wstride * es) % 16 || (span != 128 && span != 64)) return DW_ERR_ARG;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)nw};
    cuuint64_t strides[2] = {(cuuint64_t)ld * es, (cuuint64_t)wstride * es};
    cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, (cuuint32_t)box_w};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                    const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? DW_OK : DW_ERR_ARG;
}

int* tc_error_flag() {
    void* p = nullptr;
    return cudaGetSymbolAddress(&p, g_tc_error) == cudaSuccess ? static_cast<int*>(p) : nullptr;
}

int num_sms() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

namespace {

constexpr int BM = 128;
constexpr int kEpiWarps = 8;                         // two per TMEM lane quarter
constexpr int kThreads = 64 + 32 * kEpiWarps;        // producer warp, MMA warp, epilogue warps
constexpr int CW = 32;                               // columns per epilogue chunk / staged store box
constexpr int kSmemMax = 220 * 1024;                 // dynamic shared memory of a CTA at most

// named barrier 1: all epilogue warps
__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory"); }

// 16-byte chunk j of row r in a 128-byte-swizzled staging tile (128-byte rows, 1024-byte aligned).
__device__ __forceinline__ uint32_t swz(int r, int j) { return (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)); }
// 16-byte chunk j (0..3) of row r in a 64-byte-swizzled staging tile (64-byte rows): the chunk
// index is XORed with address bits 7-8, i.e. with (r >> 1) & 3.
__device__ __forceinline__ uint32_t swz64(int r, int j) { return (uint32_t)(r * 64 + ((j ^ ((r >> 1) & 3)) << 4)); }

struct TcArgs {
    int M, N, K, BN;
    GemmEpi epi;
    int stages;
    uint32_t tmem_cols;
    int n_tiles_n, n_tiles;
};

// OUT: 0 = fp32 C, 1 = bf16 C, 2 = split-BF16 C. BK: K-columns per pipeline stage (64 or 32).
template <int NP, int OUT, int BK>
__global__ void __launch_bounds__(kThreads, 1)
k_gemm_tc(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
          const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
          const __grid_constant__ CUtensorMap tmC0, const __grid_constant__ CUtensorMap tmC1, TcArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int SWB = 4096;                          // staging bytes per buffer (32 x CW fp32, or BF16 hi + lo)
    const int S = a.stages, BN = a.BN;
    const uint32_t a_bytes = BM * BK * 2, b_bytes = (uint32_t)BN * BK * 2;
    const uint32_t stage_bytes = NP * (a_bytes + b_bytes);
    auto sA = [&](int s, int part) { return smem + (size_t)s * stage_bytes + (size_t)part * a_bytes; };
    auto sB = [&](int s, int part) { return smem + (size_t)s * stage_bytes + (size_t)NP * a_bytes + (size_t)part * b_bytes; };
    uint8_t* stage_out = smem + (size_t)S * stage_bytes;                   // [epilogue warp][2 buffers][SWB]
    uint64_t* full = reinterpret_cast<uint64_t*>(stage_out + 2 * kEpiWarps * SWB);
    uint64_t* empty = full + S;
    uint64_t* tfull = empty + S;     // [2]
    uint64_t* tempty = tfull + 2;    // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    __shared__ int s_err;
    __shared__ int s_epi_err;   // written only by epilogue warps, read after their named barrier

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = (a.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        s_err = 0;
        s_epi_err = 0;
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], kEpiWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer
        if (lane == 0) {
            uint32_t cnt = 0;
            uint32_t issued[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            bool err = false;
            for (int tile = blockIdx.x; tile < a.n_tiles && !err; tile += gridDim.x) {
                const int m0 = (tile / a.n_tiles_n) * BM, n0 = (tile % a.n_tiles_n) * BN;
                for (int kt = 0; kt < nk; ++kt, ++cnt) {
                    const int s = cnt % S;
                    const uint32_t use = cnt / S;
                    if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1)) { err = true; break; }
                    mbar_expect_tx(&full[s], stage_bytes);
                    tma_load_2d(sA(s, 0), &tmA0, &full[s], kt * BK, m0);
                    if (NP == 2) tma_load_2d(sA(s, 1), &tmA1, &full[s], kt * BK, m0);
                    tma_load_2d(sB(s, 0), &tmB0, &full[s], kt * BK, n0);
                    if (NP == 2) tma_load_2d(sB(s, 1), &tmB1, &full[s], kt * BK, n0);
                    issued[s] = use + 1;
                }
            }
            if (err) {
                atomicExch(&s_err, 1);
                for (int s = 0; s < S; ++s)          // drain loads still in flight
                    if (issued[s]) mbar_wait(&full[s], (issued[s] - 1) & 1);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(BN);
            uint32_t cnt = 0, it = 0;
            bool err = false;
            for (int tile = blockIdx.x; tile < a.n_tiles && !err; tile += gridDim.x, ++it) {
                const uint32_t acc = it & 1;
                if (!mbar_wait(&tempty[acc], ((it >> 1) & 1) ^ 1)) { err = true; break; }
                tc_fence_after();
                const uint32_t d = tmem + acc * (uint32_t)BN;
                for (int kt = 0; kt < nk; ++kt, ++cnt) {
                    const int s = cnt % S;
                    if (!mbar_wait(&full[s], (cnt / S) & 1)) { err = true; break; }
                    tc_fence_after();
                    const uint64_t a0 = smem_desc<BK>(sA(s, 0)), b0 = smem_desc<BK>(sB(s, 0));
                    const uint64_t a1 = smem_desc<BK>(sA(s, NP - 1)), b1 = smem_desc<BK>(sB(s, NP - 1));
                    #pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        const uint64_t o = (uint64_t)(kk * 2);
                        umma_bf16(d, a0 + o, b0 + o, idesc, (kt | kk) ? 1u : 0u);
                        if (NP == 2) {
                            umma_bf16(d, a0 + o, b1 + o, idesc, 1u);
                            umma_bf16(d, a1 + o, b0 + o, idesc, 1u);
                        }
                    }
                    umma_commit(&empty[s]);
                }
                umma_commit(&tfull[acc]);
            }
            if (err) atomicExch(&s_err, 1);
        }
    } else {
        // ---------------- epilogue warps: warp w drains TMEM lanes 32 (w % 4) .. +31; the two warps
        // of one lane quarter take alternate CW-column chunks (column half h)
        const int q = warp & 3;                      // TMEM lane quarter
        const int ew = warp - 2, h = ew >> 2;        // epilogue warp index, column half
        const GemmEpi& e = a.epi;
        const int Tp = e.Tp;
        uint32_t nchunk = 0;                         // chunks staged by this warp (selects the buffer)
        uint32_t it = 0;
        for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x, ++it) {
            const int m0 = (tile / a.n_tiles_n) * BM, n0 = (tile % a.n_tiles_n) * BN;
            const uint32_t acc = it & 1;
            const int row = q * 32 + lane;           // row within the tile
            const int m = m0 + row;
            const int t = m % Tp;
            const float* rb = (e.rowbias && m < a.M) ? e.rowbias + ((int64_t)(m / e.rows_per_walker) * Tp + t) * e.ldrb
                                                     : nullptr;
            const bool is_val = t == 0;
            // bias / row-bias of one CW-column chunk (vectorized; rows of one walker share their
            // row-bias rows, so neighbouring warps hit in L1)
            float rbv[CW];
            auto load_bias = [&](int c0) {
                const bool full_chunk = n0 + c0 + CW <= a.N;
                #pragma unroll
                for (int j = 0; j < CW; j += 4) {
                    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                    const int n = n0 + c0 + j;
                    if (rb) {
                        if (full_chunk) x = __ldg(reinterpret_cast<const float4*>(rb + n));
                        else {
                            if (n < a.N) x.x = __ldg(rb + n);
                            if (n + 1 < a.N) x.y = __ldg(rb + n + 1);
                            if (n + 2 < a.N) x.z = __ldg(rb + n + 2);
                            if (n + 3 < a.N) x.w = __ldg(rb + n + 3);
                        }
                    }
                    if (e.bias && is_val) {
                        if (full_chunk) {
                            float4 b4 = __ldg(reinterpret_cast<const float4*>(e.bias + n));
                            x.x += b4.x; x.y += b4.y; x.z += b4.z; x.w += b4.w;
                        } else {
                            if (n < a.N) x.x += __ldg(e.bias + n);
                            if (n + 1 < a.N) x.y += __ldg(e.bias + n + 1);
                            if (n + 2 < a.N) x.z += __ldg(e.bias + n + 2);
                            if (n + 3 < a.N) x.w += __ldg(e.bias + n + 3);
                        }
                    }
                    rbv[j] = x.x; rbv[j + 1] = x.y; rbv[j + 2] = x.z; rbv[j + 3] = x.w;
                }
            };
            if (rb) {
                // pull this row's row-bias chunks into L1 while the accumulator is finished
                for (int c0 = h * CW; c0 < BN && n0 + c0 < a.N; c0 += 2 * CW)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(rb + n0 + c0));
            }
            const bool ready = mbar_wait(&tfull[acc], (it >> 1) & 1);
            if (!ready && lane == 0) s_epi_err = 1;
            epi_bar();                               // all epilogue warps agree before leaving
            if (*(volatile int*)&s_epi_err) { if (lane == 0) atomicExch(&s_err, 1); break; }
            tc_fence_after();
            for (int c0 = h * CW; c0 < BN; c0 += 2 * CW) {
                float v[CW];
                load_bias(c0);                        // issued before the TMEM reads of this chunk
                const uint32_t base = tmem + acc * (uint32_t)BN + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
                #pragma unroll
                for (int j = 0; j < CW; j += 16) tmem_ld16(base + j, v + j);
                tmem_wait_ld(v);
                #pragma unroll
                for (int j = 0; j < CW; ++j) v[j] += rbv[j];
                // double-buffered staging: the store issued from this buffer two chunks ago has
                // finished reading it once at most one bulk group (the previous chunk's) is pending
                uint8_t* my_out = stage_out + (size_t)(ew * 2 + (nchunk & 1)) * SWB;
                ++nchunk;
                if (lane == 0) bulk_wait_read1();
                __syncwarp();
                if (e.act == 1) {
                    #pragma unroll
                    for (int j = 0; j < CW; ++j) v[j] = tanhf(v[j]);
                }
                // stage the 32 x CW sub-tile (128-byte swizzle for FP32 rows, 64-byte for BF16 rows) and
                // store it with TMA
                if (OUT == 0) {
                    #pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<float4*>(my_out + swz(lane, j)) =
                            make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else {
                    #pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t hw_[4], lw_[4];
                        #pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float x0 = v[8 * j + 2 * k], x1 = v[8 * j + 2 * k + 1];
                            const __nv_bfloat162 hh = __floats2bfloat162_rn(x0, x1);
                            hw_[k] = *reinterpret_cast<const uint32_t*>(&hh);
                            if (OUT == 2) {
                                const __nv_bfloat162 ll = __floats2bfloat162_rn(x0 - __low2float(hh), x1 - __high2float(hh));
                                lw_[k] = *reinterpret_cast<const uint32_t*>(&ll);
                            } else {
                                lw_[k] = 0u;
                            }
                        }
                        *reinterpret_cast<uint4*>(my_out + swz64(lane, j)) = make_uint4(hw_[0], hw_[1], hw_[2], hw_[3]);
                        if (OUT == 2)
                            *reinterpret_cast<uint4*>(my_out + 2048 + swz64(lane, j)) = make_uint4(lw_[0], lw_[1], lw_[2], lw_[3]);
                    }
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&tmC0, my_out, n0 + c0, m0 + q * 32);
                    if (OUT == 2) tma_store_2d(&tmC1, my_out + 2048, n0 + c0, m0 + q * 32);
                    bulk_commit();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[acc]);
        }
        if (lane == 0) bulk_wait0();
    }
    tc_fence_before();
    __syncthreads();
    if (s_err && threadIdx.x == 0) atomicExch(&g_tc_error, 1);
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------ host side
// A: NP parts of a logical [M, lda] activation (NP = 2: [hi | lo] rows of width 2 lda).
// W0/W1: [N, round_up(K, 64)] K-major weight parts. C: logical [M, ldc].
// K-columns per stage of the split-BF16 GEMMs (instrumentation: dw_debug_set_gemm_bk).
int g_split_bk = 64;

template <int NP, int OUT, int BK>
int launch_tc(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C, int ldc,
              int M, int N, int K, const GemmEpi& epi, cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0) return DW_OK;
    constexpr int BN_MAX = NP == 2 ? 128 : 256;      // keeps >= 2 pipeline stages in shared memory
    int ntn = (N + BN_MAX - 1) / BN_MAX;
    int BN = round_up((N + ntn - 1) / ntn, CW);
    while (BN > BN_MAX) { ntn += 1; BN = round_up((N + ntn - 1) / ntn, CW); }
    const int Kp = round_up(K, 64);
    CUtensorMap ma0, ma1, mb0, mb1, mc0, mc1;
    DW_CHECK(make_map(&ma0, A, M, K, (int64_t)NP * lda, BK, BM, false));
    if (NP == 2) DW_CHECK(make_map(&ma1, A + lda, M, K, (int64_t)NP * lda, BK, BM, false));
    else ma1 = ma0;
    DW_CHECK(make_map(&mb0, W0, N, K, Kp, BK, BN, false));
    if (NP == 2) DW_CHECK(make_map(&mb1, W1, N, K, Kp, BK, BN, false));
    else mb1 = mb0;
    if (OUT == 0) {
        DW_CHECK(make_map(&mc0, C, M, N, ldc, 32, 32, true));
        mc1 = mc0;
    } else if (OUT == 1) {
        DW_CHECK(make_map(&mc0, C, M, N, ldc, 32, 32, false));
        mc1 = mc0;
    } else {
        DW_CHECK(make_map(&mc0, C, M, N, (int64_t)2 * ldc, 32, 32, false));
        DW_CHECK(make_map(&mc1, reinterpret_cast<const __nv_bfloat16*>(C) + ldc, M, N, (int64_t)2 * ldc, 32, 32, false));
    }
    TcArgs a;
    a.M = M; a.N = N; a.K = K; a.BN = BN; a.epi = epi;
    const int stage_bytes = NP * (BM * BK * 2 + BN * BK * 2);
    const int fixed = 1024 + 2 * kEpiWarps * 4096 + 256;
    a.stages = std::min(8, (kSmemMax - fixed) / stage_bytes);
    if (a.stages < 2) return DW_ERR_ARCH;
    a.tmem_cols = 32;
    while ((int)a.tmem_cols < 2 * BN) a.tmem_cols <<= 1;
    const int mt = (M + BM - 1) / BM;
    a.n_tiles_n = ntn;
    a.n_tiles = mt * ntn;
    size_t smem = (size_t)fixed + (size_t)a.stages * stage_bytes;
    auto kern = k_gemm_tc<NP, OUT, BK>;
    DW_CHECK_CUDA(allow_smem(kern, kSmemMax));
    int grid = std::min(a.n_tiles, num_sms());
    kern<<<grid, kThreads, smem, s>>>(ma0, ma1, mb0, mb1, mc0, mc1, a);
    count_launch();
    DW_CHECK_CUDA(launch_error());
    return DW_OK;
}

}  // namespace

bool tc_available() {
    static int cached = -1;
    if (cached < 0) {
        const char* env = getenv("DWGB_DISABLE_TC");
        int dev = 0;
        cudaDeviceProp prop;
        cached = (!(env && env[0] == '1') && cudaGetDevice(&dev) == cudaSuccess &&
                  cudaGetDeviceProperties(&prop, dev) == cudaSuccess && prop.major == 10 && prop.minor == 3 &&
                  encode_fn() != nullptr) ? 1 : 0;
    }
    return cached == 1;
}

int gemm_tc(int np, int out, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C, int ldc,
            int M, int N, int K, const GemmEpi& epi, cudaStream_t s) {
    const __nv_bfloat16* a = reinterpret_cast<const __nv_bfloat16*>(A);
    if (np == 1 && out == 0) return launch_tc<1, 0, 64>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
    if (np == 1 && out == 1) return launch_tc<1, 1, 64>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
    if (g_split_bk == 32) {
        if (np == 2 && out == 0) return launch_tc<2, 0, 32>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
        if (np == 2 && out == 2) return launch_tc<2, 2, 32>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
    }
    if (np == 2 && out == 0) return launch_tc<2, 0, 64>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
    if (np == 2 && out == 2) return launch_tc<2, 2, 64>(a, lda, W0, W1, C, ldc, M, N, K, epi, s);
    return DW_ERR_ARG;
}

}  // namespace dw

extern "C" {

// Test hook: C[M,N] (fp32) = A[M,K] (bf16, row stride lda) @ Wt[N,K]^T (bf16, row stride round_up(K,64)).
// With Wt_lo != NULL, A is split-BF16 ([hi | lo] rows of logical width lda) and W = Wt + Wt_lo.
int dw_debug_gemm_bf16(const void* A, int lda, const void* Wt, const void* Wt_lo, float* C, int ldc, int M, int N, int K,
                       void* stream) {
    if (!dw::tc_available()) return DW_ERR_UNSUPPORTED;
    dw::GemmEpi e;
    return dw::gemm_tc(Wt_lo ? 2 : 1, 0, A, lda, (const __nv_bfloat16*)Wt, (const __nv_bfloat16*)Wt_lo, C, ldc, M, N, K,
                       e, (cudaStream_t)stream);
}

// Instrumentation: K-columns per pipeline stage of the split-BF16 GEMMs (64: two stages of 64 KB at
// N tiles of 128; 32: four stages of 32 KB). Returns the previous value; other values are ignored.
int dw_debug_set_gemm_bk(int bk) {
    const int prev = dw::g_split_bk;
    if (bk == 32 || bk == 64) dw::g_split_bk = bk;
    return prev;
}

// Reads and clears the device-side error flag of the tensor-core kernels (1 = a bounded wait timed out).
int dw_debug_tc_error_flag(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, dw::g_tc_error, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(dw::g_tc_error, &zero, sizeof(int));
    return v;
}

}  // extern "C"
