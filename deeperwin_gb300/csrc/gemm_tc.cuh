// Persistent tcgen05 tensor-core GEMM (TMA loads, TMEM accumulators, TMA stores).
#pragma once
#include "net.cuh"
#include "tc_ptx.cuh"

namespace dw {

bool tc_available();
int num_sms();
int* tc_error_flag();      // device address of the error flag of the tensor-core kernels (null on failure)

// Tensor maps of K-major tiles (swizzle = box_cols * element size: 128 or 64 bytes).
int make_map(CUtensorMap* map, const void* base, int64_t rows, int cols, int64_t ld, int box_cols, int box_rows,
             bool f32);
int make_map3(CUtensorMap* map, const void* base, int64_t nw, int rows, int cols, int64_t ld, int64_t wstride,
              int box_cols, int box_rows, int box_w, bool f32);

// C[M, N] = epilogue(A[M, K] @ W[N, K]^T).
// np = 1: A and W are BF16; np = 2: split-BF16 (A is [hi | lo] rows of logical width lda, W = W0 + W1).
// out = 0: fp32 C (row stride ldc); 1: bf16 C; 2: split-BF16 C ([hi | lo] rows of logical width ldc).
// Bias / row bias and optional tanh (epi.act). W rows have stride round_up(K, 64).
int gemm_tc(int np, int out, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C, int ldc,
            int M, int N, int K, const GemmEpi& epi, cudaStream_t s);

// Rows of a tangent pass: T channel rows of electrons [i0, i0 + ns) of each of nw walkers of n electrons.
struct JetRows {
    int nw, n, T, ns, i0;
};
// C[(e, t), f] over those rows (the same rows of A and C) with bias (value rows), row bias (one row per
// walker and channel) and the forward-Laplacian tanh over each electron's T rows. np, out and the
// strides as for gemm_tc; no alignment is asked of C. T <= 128.
int gemm_jet(int np, int out, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C,
             int ldc, const JetRows& rows, int NF, int K, const GemmEpi& epi, cudaStream_t s);

// Backflow of one spin's rows times the envelope, straight into the Slater channels: features are the
// orbital columns (k, o), MO[b][k][t][i][o] = env[i, (k, o)] * bf[(b, i, t), (k, o)] with the product rule.
struct EnvEpi {
    const float* r; const float* R; const int32_t* Z;       // walkers, nuclei (per geometry segment)
    const float* sp_alpha; const float* wts;                // this spin's softplus(alpha), weights [N][KN]
    float* MO;
    Dims d;
};
int gemm_jet_env(int np, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, const JetRows& rows,
                 int K, const EnvEpi& env, cudaStream_t s);

}  // namespace dw
