// FP64 GEMM on the BF16 tensor cores by exact digit products (fp64_gemm.cu).
#pragma once
#include "net.cuh"

namespace dw {

constexpr int kDig = 9;            // signed 7-bit digits of a row- or column-scaled 62-bit fixed-point value
constexpr int kMaxK64 = 512;       // widest reduction (the spin-mean rows of a 256-wide layer)
inline int pad_k64(int K) { return round_up(K, 32); }

// Planes of one operand: dig[plane][row][Kp], kDig of digits (BF16 integers in [-64, 64]) and, for the general
// product, one of magnitudes; row exponents ex[row].
struct Digits {
    __nv_bfloat16* dig;
    int* ex;
    int64_t rows;                  // rows of a plane
    int Kp;
    int planes;
};
constexpr int planes64(bool batch) { return batch ? kDig : kDig + 1; }
// Weights [K, N] row-major FP32 (stride ldw) and their digit planes (rows = columns of W).
struct Weight64 {
    const float* w;
    int ldw, K, N;
    Digits d;
};

// Rows of a GEMM: up to two groups, each `rpw` consecutive digit rows per walker from `base` on; row
// rem of walker b is row b * out_rpw + out_off + rem of A and C.
struct RowGroup {
    int64_t base;
    int rpw;
    int64_t out_rpw, out_off;
};
struct Rows64 {
    int ngroups;
    RowGroup g[2];
    int B;                         // walkers
    const int* nvalid;             // device-side walker count (null: B); valid are *nvalid mul - first
    int mul = 1, first = 0;
};
inline Rows64 plain_rows(int B, int rpw, const int* nvalid) {
    Rows64 r;
    r.ngroups = 1; r.B = B; r.nvalid = nvalid;
    r.g[0] = r.g[1] = RowGroup{0, rpw, rpw, 0};
    return r;
}

// Digit planes of the rows of A [.., K] (row stride lda); skips walkers beyond nvalid.
void slice_rows64(const double* A, int lda, int K, const Rows64& rows, const Digits& d, cudaStream_t s);
// Spin means M [(b, t)][2 hw] of X's first hw columns over the nu up and n - nu down electrons, and their digit planes
// (none if d.dig is null).
void spin_means64(const double* X, int ldx, int hw, int n, int nu, int C, const Rows64& rows, double* M, const Digits& d,
                  cudaStream_t s);
// Digit planes of `count` weight matrices in one launch (nothing when *nvalid == 0).
constexpr int kMaxW64 = 16;
void slice_weights64(const Weight64* w, int count, const int* nvalid, cudaStream_t s);

// C[m, n] = sum_k A[m, k] W[k, n] (+ bias[n] on rows whose channel, row % C, is 0) (+ rowbias[(walker,
// channel), n]). A is the FP64 matrix the digits were cut from.
struct Epi64 {
    const float* bias = nullptr;
    const double* rowbias = nullptr;
    int ldrb = 0;
};
// FP64 determinant tangents of nmat matrices with T - 1 derivative channels (MO64 [mat][T][n][n], Ainv64
// [mat][n][n], sign): g[mat][3 n] = tr(A^-1 dA_t), lapdet[mat] = tr(A^-1 Lap A) - sum_t tr((A^-1 dA_t)^2), as
// digit products. K determinants per walker (nvalid counts walkers, these start at `first`). Returns false, having done nothing,
// where the FP64 loop is as fast (n < 24), for n > 48, or with scratch for less than 32 matrices at a time.
size_t dets64_scratch_bytes(int n, int T, int64_t nmat);
bool dets64_tangents(const double* MO64, const double* Ainv64, const double* sign, int n, int T, int K, int nmat,
                     const int* nvalid, int first, double* g, double* lapdet, void* scratch, size_t scratch_bytes, cudaStream_t s,
                     int* status);

// The product by digits (A's planes da, w.d).
int gemm64_tc(const double* A, int lda, const Digits& da, const Weight64& w, double* C, int ldc, const Rows64& rows,
              int channels, const Epi64& e, cudaStream_t s);
// The product on the FP64 pipe, for workspaces without room for the planes.
int gemm64_pipe(const double* A, int lda, const Weight64& w, double* C, int ldc, const Rows64& rows, int channels,
                const Epi64& e, cudaStream_t s);

}  // namespace dw
