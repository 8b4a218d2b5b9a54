// FP64 matrix product on the BF16 tensor cores, by splitting both operands into small integers
// (K. Ozaki, T. Ogita, S. Oishi, S. Rump, "Error-free transformations of matrix multiplication by
// using fast routines of matrix multiplication and its applications", Numer. Algorithms 59, 2012; on
// tensor cores: D. Mukunoki et al., "DGEMM using tensor cores, and its accurate and reproducible
// versions", ISC 2020).
//
// Each row of A and each column of W is scaled by a power of two so that its largest magnitude is
// below one, rounded to 62 fractional bits and written as nine signed 7-bit digits,
//   a = 2^Ea sum_i d_i 2^(-6 - 7 i),  d_0 in [-64, 64], d_i in [-64, 63].
// A digit is exact in BF16, a product of two digits is below 2^12, and the sum of the up to nine
// products with i + j = s over K <= 512 columns stays below 2^24 (for s = 8 and K = 512 the bound is
// 2^24.2, reached only if every digit were extreme; a rounding there is 2^-56 of the last digit), so
// the FP32 accumulators in TMEM hold every digit sum exactly, in any order. The 45 products with
// i + j <= 8 give the result to about 2^-61 sqrt(K) max|a| max|w| (at most K 2^-59.5); the nine sums
// are combined in integers and rounded to FP64 once. FP32 weights are represented exactly down to
// 2^-38 of their column's maximum.
//
// The error of an FP64 sum is relative to S = sum |a| |w| instead, which is far below max|a| max|w| where
// large entries of a row meet small entries of a column. A tenth plane of each operand therefore holds the
// magnitudes |a| 2^-Ea in BF16, whose product is S to 1 %: outputs with S below 2^-6 of both scales
// (kTrust) are formed by an FP64 sum over the original values, so every output is within K 2^-53 S. Rows and
// columns of zeros give zero. (Determinants, BATCH, balance their inner index instead, see dets64_tangents.)
// Layers' rows have S far above that, so the sum is rare; the plane is 1 MMA in 46 and a tenth of the bytes (FP64
// form, C2H4, 64 walkers: 9.93 -> 10.08 ms).
//
// Why: FP64 issues at about two lanes per clock and SM here (1.2 TFLOP/s), the BF16 tensor cores at
// about 1500 times that, so even 45 products per multiplication are far cheaper: the 16 GEMMs of a
// C2H4-shaped local energy (16 electrons, 32 determinants, 64 walkers) took 46.0 ms on the FP64 pipe
// (64 x 64 tiles, 0.97 TFLOP/s) and take 4.7 ms here; a single tile of the FP64 loop takes longer than
// the smallest launch of this kernel, so no size keeps it. It serves workspaces without room for the planes.
//
// Rows and columns whose scale is not an ordinary one (infinities, NaN, below 2^-922) are computed
// from the original FP64 values in the epilogue.
#include "fp64_gemm.cuh"
#include "gemm_tc.cuh"
#include <algorithm>

namespace dw {

namespace {

constexpr int BM = 128, BN = 48, BK = 32;            // rows, columns, K-columns of a pipeline stage
constexpr int kStages = 2;
constexpr int kEpi = 8;                              // epilogue warps: two per TMEM lane quarter
constexpr int kThreads64 = 64 + 32 * kEpi;
constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2;      // one plane of a stage
constexpr int stage_bytes64(int planes) { return planes * (kABytes + kBBytes); }
constexpr int smem64(int planes) { return 1024 + kStages * stage_bytes64(planes) + 256; }
constexpr int kFlagged = 0x7fffffff;                 // exponent of a row that the digits do not represent
constexpr int kZeroRow = -0x7fffffff;                // of a row of zeros
constexpr float kTrust = 1.0f / 64;

__device__ __forceinline__ int valid_of(const Rows64& r) { return r.nvalid ? min(r.B, max(0, *r.nvalid * r.mul - r.first)) : r.B; }

// Biased exponent field of x.
__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// What a row's exponent E follows from (values are below 2^E): the largest exponent field, here of unscaled
// entries. Subnormal entries have no digits, so the largest has to be far above them.
struct RowScan {
    int emax = 0;
    uint32_t any = 0;
    __device__ __forceinline__ void add(double x) {
        emax = max(emax, exp_field(x));
        any |= (uint32_t)__double2loint(x) | ((uint32_t)__double2hiint(x) << 1);
    }
    __device__ __forceinline__ int exponent() const {
        if (emax == 0) return any ? kFlagged : kZeroRow;
        return emax == 0x7ff || emax < 100 ? kFlagged : emax - 1022;
    }
    __device__ __forceinline__ int merge_warp() {
        emax = __reduce_max_sync(0xffffffffu, emax);
        any = __any_sync(0xffffffffu, any != 0);
        return exponent();
    }
};
// The same of entries taken times 2^shift: the field may leave its range, subnormal entries and infinities are
// kept apart.
struct ScaledRowScan {
    static constexpr int kNone = -(1 << 20);
    int emax = kNone, sub = kNone, special = 0;
    __device__ __forceinline__ void add(double x, int shift) {
        const long long bits = __double_as_longlong(x);
        const int e = (int)(bits >> 52) & 0x7ff;
        if (e == 0x7ff) special = 1;
        else if (e) emax = max(emax, e + shift);
        else if (bits << 1) sub = max(sub, 1 + shift);
    }
    __device__ __forceinline__ int merge_warp() {
        emax = __reduce_max_sync(0xffffffffu, emax);
        sub = __reduce_max_sync(0xffffffffu, sub);
        special = __reduce_max_sync(0xffffffffu, special);
        if (special || (sub != kNone && sub > emax - 64)) return kFlagged;
        return emax == kNone ? kZeroRow : emax - 1022;
    }
};
// x 2^(62 - E) rounded to an integer (E = emax - 1022), |result| <= 2^62.
__device__ __forceinline__ long long to_fixed(double x, int emax) {
    const long long bits = __double_as_longlong(x);
    const int e = (int)(bits >> 52) & 0x7ff;
    unsigned long long m = (bits & 0xfffffffffffffll) | (1ll << 52);
    const int sh = emax - e - 9;             // right shift of the 53-bit significand
    if (e == 0 || sh > 54) return 0;
    m = sh <= 0 ? m << -sh : (m + (1ull << (sh - 1))) >> sh;
    return bits < 0 ? -(long long)m : (long long)m;
}
// Next digit from the low end: d in [-64, 63], x <- (x - d) / 128.
__device__ __forceinline__ int low_digit(long long& x) {
    const int d = (((int)x & 127) ^ 64) - 64;
    x = (x - d) >> 7;
    return d;
}
__device__ __forceinline__ uint32_t pack_digits(int a, int b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn((float)a, (float)b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Magnitudes of two fixed-point values (62 fractional bits).
__device__ __forceinline__ uint32_t pack_magnitudes(long long a, long long b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn((float)(a < 0 ? -a : a) * 0x1p-62f, (float)(b < 0 ? -b : b) * 0x1p-62f);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// One row held by a warp (columns 64 u + 2 lane, + 1) of exponent E: its planes. emax(u, k): largest exponent field
// of the row less the shift of column 64 u + 2 lane + k.
template <int NU, class EMax>
__device__ __forceinline__ void slice_row(const double2 (&x)[NU], int E, EMax emax, int64_t m, const Digits& d) {
    const int lane = threadIdx.x & 31, Kp = d.Kp;
    if (lane == 0) d.ex[m] = E;
    __nv_bfloat16* o = d.dig + m * Kp;
    const int64_t plane = d.rows * Kp;
    #pragma unroll
    for (int u = 0; u < NU; ++u) {
        const int c = u * 64 + 2 * lane;
        if (c >= Kp) continue;
        long long f0 = 0, f1 = 0;
        if (E != kFlagged) { f0 = to_fixed(x[u].x, emax(u, 0)); f1 = to_fixed(x[u].y, emax(u, 1)); }
        if (d.planes > kDig) *reinterpret_cast<uint32_t*>(o + kDig * plane + c) = pack_magnitudes(f0, f1);
        #pragma unroll
        for (int i = kDig - 1; i >= 0; --i) {
            const int d0 = i ? low_digit(f0) : (int)f0, d1 = i ? low_digit(f1) : (int)f1;
            *reinterpret_cast<uint32_t*>(o + i * plane + c) = pack_digits(d0, d1);
        }
    }
}

// Warp per row: the largest exponent, then the digits of two neighbouring columns per lane and step.
// HBM-bound: 8 K bytes read, 20 Kp (BATCH: 18 Kp) written per row.
// es: distance of a row's elements; NU: groups of 64 columns. bal (BATCH): exponents [matrix][K] by which the
// columns are scaled, times 2^(sign bal).
template <int NU, bool BATCH>
__global__ void __launch_bounds__(256)
k64_slice_rows(const double* __restrict__ A, int lda, int es, int K, Rows64 rows, const int* __restrict__ bal, int sign,
               Digits d) {
    const int nv = valid_of(rows), lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int gi = rows.ngroups > 1 && w >= (int64_t)rows.B * rows.g[0].rpw ? 1 : 0;
    const RowGroup& g = rows.g[gi];
    const int64_t k = gi ? w - (int64_t)rows.B * rows.g[0].rpw : w;    // row within the group
    const int64_t b = k / g.rpw;
    if (b >= nv) return;
    const int64_t m = g.base + k;
    const double* src = A + (b * g.out_rpw + g.out_off + k % g.rpw) * lda;
    double2 x[NU];
    #pragma unroll
    for (int u = 0; u < NU; ++u) {
        const int c = u * 64 + 2 * lane;
        x[u] = make_double2(0.0, 0.0);
        if (c < K) x[u].x = src[(int64_t)c * es];
        if (c + 1 < K) x[u].y = src[(int64_t)(c + 1) * es];
    }
    if constexpr (BATCH) {
        int shift[NU][2];
        ScaledRowScan scan;
        #pragma unroll
        for (int u = 0; u < NU; ++u)
            #pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int c = u * 64 + 2 * lane + v;
                shift[u][v] = c < K ? sign * bal[b * K + c] : 0;
                scan.add(v ? x[u].y : x[u].x, shift[u][v]);
            }
        const int E = scan.merge_warp();
        slice_row(x, E, [&](int u, int v) { return scan.emax - shift[u][v]; }, m, d);
    } else {
        RowScan scan;
        #pragma unroll
        for (int u = 0; u < NU; ++u) { scan.add(x[u].x); scan.add(x[u].y); }
        const int E = scan.merge_warp();
        slice_row(x, E, [&](int, int) { return scan.emax; }, m, d);
    }
}

// Exponents bal[matrix][o] of the rows of W (largest entry in [2^bal, 2^(bal + 1)); 0 for rows without an
// ordinary one), warp per row.
__global__ void __launch_bounds__(256)
k64_balance(const double* __restrict__ W, int n, Rows64 rows, int* __restrict__ bal) {
    const int row = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (row / n >= valid_of(rows)) return;
    int e = 0;
    for (int c = lane; c < n; c += 32) e = max(e, exp_field(W[(int64_t)row * n + c]));
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) bal[row] = e == 0 || e == 0x7ff ? 0 : e - 1023;
}

// Spin means of the hw columns of X per (walker, channel), M[(b, t)] = [mean over up electrons, mean
// over down electrons] (SymmetricFeatures, ferminet_embedding.py:52-94), and their digit planes; warp
// per row of M.
__global__ void __launch_bounds__(256)
k64_spin_means(const double* __restrict__ X, int ldx, int hw, int n, int nu, int C, Rows64 rows, double* __restrict__ M,
               Digits d) {
    const int64_t bt = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t b = bt / C;
    if (b >= valid_of(rows)) return;
    const int t = (int)(bt % C), lane = threadIdx.x & 31;
    double2 x[kMaxK64 / 64];
    RowScan scan;
    #pragma unroll
    for (int u = 0; u < kMaxK64 / 64; ++u) {
        double v[2] = {0.0, 0.0};
        #pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int c = u * 64 + 2 * lane + k;
            if (c >= 2 * hw) continue;
            const int i0 = c < hw ? 0 : nu, i1 = c < hw ? nu : n, col = c < hw ? c : c - hw;
            double acc = 0.0;
            for (int i = i0; i < i1; ++i) acc += X[((b * n + i) * C + t) * (int64_t)ldx + col];
            v[k] = acc / (i1 - i0);
            M[bt * 2 * hw + c] = v[k];
            scan.add(v[k]);
        }
        x[u] = make_double2(v[0], v[1]);
    }
    if (!d.dig) return;
    const int E = scan.merge_warp();
    slice_row(x, E, [&](int, int) { return scan.emax; }, bt, d);
}

struct WeightTable {
    Weight64 w[kMaxW64];
    int first[kMaxW64 + 1];                           // first block of each matrix (32 columns per block)
    int count;
    const int* nvalid;
};

// Block per 32 columns of a weight matrix: column exponents, then digits by 64-row tiles transposed
// through shared memory so that a warp writes consecutive K.
__global__ void __launch_bounds__(256) k64_slice_weights(WeightTable t) {
    if (t.nvalid && *t.nvalid <= 0) return;
    int mi = 0;
    while (mi + 1 < t.count && (int)blockIdx.x >= t.first[mi + 1]) ++mi;
    const Weight64& w = t.w[mi];
    const int n0 = ((int)blockIdx.x - t.first[mi]) * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    __shared__ float tile[64][33];
    __shared__ int emax_s[8][32];
    RowScan scan;                                     // (an FP32 value is never subnormal in FP64)
    if (n0 + tx < w.N)
        for (int k = ty; k < w.K; k += 8) scan.add((double)w.w[(int64_t)k * w.ldw + n0 + tx]);
    emax_s[ty][tx] = scan.emax;
    __syncthreads();
    if (ty == 0) {
        for (int k = 1; k < 8; ++k) scan.emax = max(scan.emax, emax_s[k][tx]);
        emax_s[0][tx] = scan.emax;
        scan.any = 0;                                 // no field: a column of zeros
        if (n0 + tx < w.N) w.d.ex[n0 + tx] = scan.exponent();
    }
    const int64_t plane = w.d.rows * w.d.Kp;
    for (int k0 = 0; k0 < w.d.Kp; k0 += 64) {
        __syncthreads();
        for (int k = ty; k < 64; k += 8)
            tile[k][tx] = k0 + k < w.K && n0 + tx < w.N ? w.w[(int64_t)(k0 + k) * w.ldw + n0 + tx] : 0.f;
        __syncthreads();
        const int k = k0 + 2 * tx;
        for (int n = ty; n < 32; n += 8) {
            if (n0 + n >= w.N || k >= w.d.Kp) continue;
            const int em = emax_s[0][n];
            const bool ok = em != 0x7ff;
            long long f0 = ok ? to_fixed((double)tile[2 * tx][n], em) : 0, f1 = ok ? to_fixed((double)tile[2 * tx + 1][n], em) : 0;
            __nv_bfloat16* o = w.d.dig + (int64_t)(n0 + n) * w.d.Kp + k;
            *reinterpret_cast<uint32_t*>(o + kDig * plane) = pack_magnitudes(f0, f1);
            #pragma unroll
            for (int i = kDig - 1; i >= 0; --i) {
                const int d0 = i ? low_digit(f0) : (int)f0, d1 = i ? low_digit(f1) : (int)f1;
                *reinterpret_cast<uint32_t*>(o + i * plane) = pack_digits(d0, d1);
            }
        }
    }
}

struct Args64 {
    const double* A; int lda;
    const float* W; int ldw;
    double* C; int ldc;
    const int* ea; const int* ew;
    Rows64 rows;
    Epi64 e;
    int N, K, channels, ntn;
    // batched form (determinants): `per` rows and N columns per matrix, W FP64 [matrix][K][N]
    const double* W64;
    int per;
    int* error;                    // set when a bounded wait ran out
};

// 2^scale sum_s acc_s 2^(56 - 7 s), rounded to the nearest double. |sum| < 2^79.
__device__ __forceinline__ double combine_digits(const float* acc, int stride, int scale) {
    long long hi = 0, lo = 0;
    #pragma unroll
    for (int s = 0; s < 4; ++s) hi = (hi << 7) + (long long)(int)acc[s * stride];
    #pragma unroll
    for (int s = 4; s < kDig; ++s) lo = (lo << 7) + (long long)(int)acc[s * stride];
    hi += lo >> 35;                                   // value = hi 2^35 + lo, 0 <= lo < 2^35
    lo &= (1ll << 35) - 1;
    const bool neg = hi < 0;
    if (neg) {
        hi = -hi;
        if (lo) { hi -= 1; lo = (1ll << 35) - lo; }
    }
    // significand with its top bit at 63, value = m 2^(e - 63)
    unsigned long long m;
    int e;
    if (hi == 0) {
        if (lo == 0) return 0.0;
        const int z = __clzll(lo);
        m = (unsigned long long)lo << z;
        e = 63 - z;
    } else {
        const int z = __clzll(hi);                    // hi < 2^45: z >= 19
        m = (unsigned long long)hi << z;
        m |= z >= 35 ? (unsigned long long)lo << (z - 35) : (unsigned long long)lo >> (35 - z);
        e = 98 - z;
    }
    unsigned long long q = m >> 11;                   // 53 bits, round to nearest even
    const unsigned rem = (unsigned)m & 0x7ffu;
    q += rem > 0x400u || (rem == 0x400u && (q & 1u));
    q += (unsigned long long)(e + scale + 1022) << 52;
    return __longlong_as_double((long long)(q | (neg ? 1ull << 63 : 0ull)));
}

// Persistent: one CTA per SM loops over 128 x 48 output tiles. Warp 0 loads the planes of 32 K-columns of
// both operands per stage (two TMA copies, 113 KB, two stages), warp 1 issues the 92 MMAs of a stage
// into ten TMEM accumulators (480 columns), eight warps combine and store them. Bound
// by the MMAs' shared-memory reads of A (N = 48: 32 clocks of reads for 24 of products); the
// accumulators leave no room for a second set, so the epilogue (about a fifth) is not overlapped.
// BATCH: each matrix has its own weights (rows [matrix N, + N) of their digit planes) and whole tiles; no
// plane of magnitudes.
template <bool BATCH>
__global__ void __launch_bounds__(kThreads64, 1)
k64_gemm_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, Args64 a) {
    constexpr int kPl = planes64(BATCH), kStageBytes = stage_bytes64(kPl);
    const int nv = valid_of(a.rows);
    int64_t tiles_of[2] = {0, 0};
    const int tpm = BATCH ? (a.per + BM - 1) / BM : 1;          // tiles per matrix
    if (BATCH) tiles_of[0] = (int64_t)nv * tpm;
    else
        for (int g = 0; g < a.rows.ngroups; ++g) tiles_of[g] = ((int64_t)nv * a.rows.g[g].rpw + BM - 1) / BM * a.ntn;
    const int64_t n_tiles = tiles_of[0] + tiles_of[1];
    if ((int64_t)blockIdx.x >= n_tiles) return;       // before any barrier or TMEM allocation
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* tfull = empty + kStages;
    uint64_t* tempty = tfull + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 1);
    __shared__ int s_err, s_epi_err;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = (a.K + BK - 1) / BK;
    if (threadIdx.x == 0) {
        s_err = 0;
        s_epi_err = 0;
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(tfull, 1);
        mbar_init(tempty, kEpi);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // tile -> row group, first row within the group, first column
    // (BATCH: the matrix, first row within it)
    auto locate = [&](int64_t tile, int& g, int64_t& k0, int& n0) {
        if (BATCH) {
            g = (int)(tile / tpm);
            k0 = tile % tpm * BM;
            n0 = 0;
            return;
        }
        g = tile >= tiles_of[0] ? 1 : 0;
        const int64_t u = g ? tile - tiles_of[0] : tile;
        k0 = u / a.ntn * BM;
        n0 = (int)(u % a.ntn) * BN;
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t cnt = 0, issued[kStages] = {0, 0};
            bool err = false;
            for (int64_t tile = blockIdx.x; tile < n_tiles && !err; tile += gridDim.x) {
                int g, n0;
                int64_t k0;
                locate(tile, g, k0, n0);
                const int row = BATCH ? (int)(g * a.per + k0) : (int)(a.rows.g[g].base + k0);
                const int wrow = BATCH ? g * a.N : n0;
                for (int kt = 0; kt < nk; ++kt, ++cnt) {
                    const int s = cnt % kStages;
                    const uint32_t use = cnt / kStages;
                    if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1)) { err = true; break; }
                    mbar_expect_tx(&full[s], kStageBytes);
                    uint8_t* st = smem + s * kStageBytes;
                    tma_load_3d(st, &tmA, &full[s], kt * BK, row, 0);
                    tma_load_3d(st + kPl * kABytes, &tmB, &full[s], kt * BK, wrow, 0);
                    issued[s] = use + 1;
                }
            }
            if (err) {
                atomicExch(&s_err, 1);
                for (int s = 0; s < kStages; ++s)
                    if (issued[s]) mbar_wait(&full[s], (issued[s] - 1) & 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(BN);
            uint32_t cnt = 0, it = 0;
            bool err = false;
            for (int64_t tile = blockIdx.x; tile < n_tiles && !err; tile += gridDim.x, ++it) {
                if (!mbar_wait(tempty, (it & 1) ^ 1)) { err = true; break; }
                tc_fence_after();
                for (int kt = 0; kt < nk; ++kt, ++cnt) {
                    const int s = cnt % kStages;
                    if (!mbar_wait(&full[s], (cnt / kStages) & 1)) { err = true; break; }
                    tc_fence_after();
                    const uint64_t da = smem_desc_sw64(smem + s * kStageBytes);
                    const uint64_t db = smem_desc_sw64(smem + s * kStageBytes + kPl * kABytes);
                    const int nkk = BATCH ? min(BK / 16, (a.K - kt * BK + 15) / 16) : BK / 16;   // 16-column steps with data
                    for (int kk = 0; kk < nkk; ++kk) {
                        if (!BATCH)
                            umma_bf16(tmem + kDig * BN, da + (uint64_t)((kDig * kABytes + kk * 32) >> 4),
                                      db + (uint64_t)((kDig * kBBytes + kk * 32) >> 4), idesc, (kt | kk) ? 1u : 0u);
                        #pragma unroll
                        for (int i = 0; i < kDig; ++i) {
                            #pragma unroll
                            for (int j = 0; j < kDig - i; ++j)
                                umma_bf16(tmem + (i + j) * BN, da + (uint64_t)((i * kABytes + kk * 32) >> 4),
                                          db + (uint64_t)((j * kBBytes + kk * 32) >> 4), idesc, (kt | kk | i) ? 1u : 0u);
                        }
                    }
                    umma_commit(&empty[s]);
                }
                umma_commit(tfull);
            }
            if (err) atomicExch(&s_err, 1);
        }
    } else {
        const int q = warp & 3, h = (warp - 2) >> 2;          // TMEM lane quarter, column half
        uint32_t it = 0;
        for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++it) {
            int g, n0;
            int64_t k0;
            locate(tile, g, k0, n0);
            const RowGroup& rg = a.rows.g[BATCH ? 0 : g];
            const int64_t k = k0 + q * 32 + lane;             // row within the group (matrix)
            const bool live = k < (BATCH ? (int64_t)a.per : (int64_t)nv * rg.rpw);
            const int64_t b = BATCH ? g : (live ? k / rg.rpw : 0);
            const int64_t rem = live ? k - (BATCH ? 0 : b * rg.rpw) : 0;
            const int64_t row = b * rg.out_rpw + rg.out_off + rem;              // of A
            const int64_t crow = BATCH ? b * a.per + rem : row;                 // of C
            const int t = (int)(row % a.channels);
            const int ea = live ? a.ea[BATCH ? crow : rg.base + k] : 0;
            const double* rb = a.e.rowbias ? a.e.rowbias + (b * a.channels + t) * a.e.ldrb : nullptr;
            const bool ready = mbar_wait(tfull, it & 1);
            if (!ready && lane == 0) s_epi_err = 1;
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");   // all epilogue warps agree
            if (*(volatile int*)&s_epi_err) { if (lane == 0) atomicExch(&s_err, 1); break; }
            tc_fence_after();
            for (int c0 = h * 8; c0 < BN; c0 += 16) {
                if (n0 + c0 >= a.N) break;
                float acc[kPl * 8];
                #pragma unroll
                for (int s = 0; s < kPl; ++s) tmem_ld8(tmem + s * BN + ((uint32_t)(q * 32) << 16) + c0, acc + s * 8);
                tmem_wait_ld(acc);
                if (live) {
                    #pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        double v[2];
                        #pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int n = min(n0 + c0 + j + u, a.N - 1);
                            const int ew = a.ew[BATCH ? g * a.N + n : n];
                            const bool flagged = ea == kFlagged || ew == kFlagged, zero = ea == kZeroRow || ew == kZeroRow;
                            const int scale = flagged || zero ? 0 : ea + ew - 68;
                            const bool trusted = BATCH || acc[(kPl - 1) * 8 + j + u] >= kTrust;
                            if (zero && !flagged) {
                                v[u] = 0.0;
                            } else if (flagged || !trusted || scale < -900 || scale > 900) {
                                double x = 0.0;
                                for (int kk = 0; kk < a.K; ++kk)
                                    x = fma(a.A[row * a.lda + kk], BATCH ? a.W64[((int64_t)g * a.K + kk) * a.N + n]
                                                                             : (double)a.W[(int64_t)kk * a.ldw + n], x);
                                v[u] = x;
                            } else {
                                v[u] = combine_digits(acc + j + u, 8, scale);
                            }
                            if (a.e.bias && t == 0) v[u] += (double)a.e.bias[n];
                            if (rb) v[u] += rb[n];
                        }
                        const int n = n0 + c0 + j;
                        double* o = a.C + crow * a.ldc + n;
                        if (n + 1 < a.N && !(a.ldc & 1)) *reinterpret_cast<double2*>(o) = make_double2(v[0], v[1]);
                        else {
                            if (n < a.N) o[0] = v[0];
                            if (n + 1 < a.N) o[1] = v[1];
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_err && threadIdx.x == 0) atomicExch(a.error, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// The same product on the FP64 pipe: 64 x 64 tiles, 16-deep K slices, 256 threads with a 4 x 4 patch each
// (rows tr + 16 i, columns tc + 16 j: a warp's shared reads of W are 16 consecutive doubles, those of A two
// broadcasts). Bound by the pipe, two lanes per clock and SM. blockIdx.z: row group.
__global__ void __launch_bounds__(256) k64_gemm_pipe(Args64 a) {
    constexpr int PM = 64, PN = 64, PK = 16;
    const RowGroup& g = a.rows.g[blockIdx.z];
    const int64_t total = (int64_t)valid_of(a.rows) * g.rpw, m0 = (int64_t)blockIdx.y * PM;
    if (m0 >= total) return;
    __shared__ double As[PK][PM + 1];
    __shared__ double Ws[PK][PN];
    __shared__ int64_t row_of[PM];
    const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16, n0 = blockIdx.x * PN;
    if (tid < PM) {
        const int64_t k = m0 + tid, b = k / g.rpw;
        row_of[tid] = k < total ? b * g.out_rpw + g.out_off + k % g.rpw : -1;
    }
    __syncthreads();
    double acc[4][4];
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        #pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    for (int k0 = 0; k0 < a.K; k0 += PK) {
        #pragma unroll
        for (int u = 0; u < PM * PK / 256; ++u) {
            const int e = tid + u * 256, r = e / PK, k = e % PK;
            As[k][r] = row_of[r] >= 0 && k0 + k < a.K ? a.A[row_of[r] * a.lda + k0 + k] : 0.0;
        }
        #pragma unroll
        for (int u = 0; u < PK * PN / 256; ++u) {
            const int e = tid + u * 256, k = e / PN, c = e % PN;
            Ws[k][c] = k0 + k < a.K && n0 + c < a.N ? (double)a.W[(int64_t)(k0 + k) * a.ldw + n0 + c] : 0.0;
        }
        __syncthreads();
        #pragma unroll
        for (int k = 0; k < PK; ++k) {
            double x[4], w[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = As[k][tr + 16 * i];
            #pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[k][tc + 16 * j];
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(x[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t row = row_of[tr + 16 * i];
        if (row < 0) continue;
        const int t = (int)(row % a.channels);
        const double* rb = a.e.rowbias ? a.e.rowbias + ((m0 + tr + 16 * i) / g.rpw * a.channels + t) * a.e.ldrb : nullptr;
        #pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tc + 16 * j;
            if (n >= a.N) continue;
            double v = acc[i][j];
            if (a.e.bias && t == 0) v += (double)a.e.bias[n];
            if (rb) v += rb[n];
            a.C[row * a.ldc + n] = v;
        }
    }
}

// Traces of E = dA_t A^-1 (cyclic: those of A^-1 dA_t), block per (matrix, channel): tr E to g (tr1 for the
// Laplacian channel), tr E^2 to tr2.
__global__ void __launch_bounds__(128)
k64_traces(const double* __restrict__ E, const double* __restrict__ sign, int n, int C, Rows64 rows, double* __restrict__ g,
           double* __restrict__ tr1, double* __restrict__ tr2) {
    const int mat = blockIdx.x / C, t = blockIdx.x % C;            // C = T - 1 channels: gradients, Laplacian
    if (mat >= valid_of(rows)) return;
    extern __shared__ double es[];                                  // [n][n + 1]
    __shared__ double red[2][4];
    const int tid = threadIdx.x, nn = n * n;
    const double* src = E + ((int64_t)mat * C + t) * nn;
    for (int e = tid; e < nn; e += 128) es[e / n * (n + 1) + e % n] = src[e];
    __syncthreads();
    double s1 = 0.0, s2 = 0.0;
    for (int e = tid; e < nn; e += 128) {
        const int i = e / n, j = e % n;
        const double x = es[i * (n + 1) + j];
        if (i == j) s1 += x;
        s2 = fma(x, es[j * (n + 1) + i], s2);
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (tid % 32 == 0) { red[0][tid / 32] = s1; red[1][tid / 32] = s2; }
    __syncthreads();
    if (tid == 0) {
        const bool ok = sign[mat] != 0.0;
        s1 = ok ? red[0][0] + red[0][1] + red[0][2] + red[0][3] : 0.0;
        if (t < C - 1) g[(int64_t)mat * (C - 1) + t] = s1;
        else tr1[mat] = s1;
        tr2[(int64_t)mat * C + t] = ok ? red[1][0] + red[1][1] + red[1][2] + red[1][3] : 0.0;
    }
}
// lapdet = tr E_lap - sum over the gradient channels of tr E_t^2, warp per matrix.
__global__ void k64_lapdet(const double* __restrict__ tr1, const double* __restrict__ tr2, int C, Rows64 rows,
                           double* __restrict__ lapdet) {
    const int mat = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (mat >= valid_of(rows)) return;
    double s = 0.0;
    for (int t = lane; t < C - 1; t += 32) s += tr2[(int64_t)mat * C + t];
    s = warp_sum(s);
    if (lane == 0) lapdet[mat] = tr1[mat] - s;
}

}  // namespace

void slice_rows64(const double* A, int lda, int K, const Rows64& rows, const Digits& d, cudaStream_t s) {
    int64_t n = 0;
    for (int g = 0; g < rows.ngroups; ++g) n += (int64_t)rows.B * rows.g[g].rpw;
    const unsigned grid = (unsigned)((n + 7) / 8);
    if (d.Kp <= 64) k64_slice_rows<1, false><<<grid, 256, 0, s>>>(A, lda, 1, K, rows, nullptr, 0, d);
    else k64_slice_rows<kMaxK64 / 64, false><<<grid, 256, 0, s>>>(A, lda, 1, K, rows, nullptr, 0, d);
    count_launch();
}

void spin_means64(const double* X, int ldx, int hw, int n, int nu, int C, const Rows64& rows, double* M, const Digits& d,
                  cudaStream_t s) {
    k64_spin_means<<<(unsigned)(((int64_t)rows.B * C + 7) / 8), 256, 0, s>>>(X, ldx, hw, n, nu, C, rows, M, d);
    count_launch();
}

void slice_weights64(const Weight64* w, int count, const int* nvalid, cudaStream_t s) {
    WeightTable t;
    t.count = count;
    t.nvalid = nvalid;
    t.first[0] = 0;
    for (int k = 0; k < count; ++k) {
        t.w[k] = w[k];
        t.first[k + 1] = t.first[k] + (w[k].N + 31) / 32;
    }
    k64_slice_weights<<<t.first[count], 256, 0, s>>>(t);
    count_launch();
}

// Multiply-adds (two operations each) of the rows' walkers, as the timers count them.
static double flops_of(const Rows64& rows, const Weight64& w) {
    double m = 0.0;
    for (int g = 0; g < rows.ngroups; ++g) m += (double)rows.B * rows.g[g].rpw;
    return 2.0 * m * w.N * w.K;
}

int gemm64_tc(const double* A, int lda, const Digits& da, const Weight64& w, double* C, int ldc, const Rows64& rows,
              int channels, const Epi64& e, cudaStream_t s) {
    if (w.K > kMaxK64 || da.Kp < w.K || w.d.Kp < w.K) return DW_ERR_ARG;
    CUtensorMap ma, mb;
    constexpr int kPl = planes64(false);
    DW_CHECK(make_map3(&ma, da.dig, kPl, (int)da.rows, da.Kp, da.Kp, da.rows * da.Kp, BK, BM, kPl, false));
    DW_CHECK(make_map3(&mb, w.d.dig, kPl, w.N, w.d.Kp, w.d.Kp, w.d.rows * w.d.Kp, BK, BN, kPl, false));
    Args64 a;
    a.A = A; a.lda = lda; a.W = w.w; a.ldw = w.ldw; a.C = C; a.ldc = ldc;
    a.ea = da.ex; a.ew = w.d.ex;
    a.rows = rows; a.e = e;
    a.N = w.N; a.K = w.K; a.channels = channels;
    a.W64 = nullptr; a.per = 0;
    a.ntn = (w.N + BN - 1) / BN;
    a.error = tc_error_flag();
    if (!a.error) return DW_ERR_CUDA;
    int64_t tiles = 0;
    for (int g = 0; g < rows.ngroups; ++g) tiles += ((int64_t)rows.B * rows.g[g].rpw + BM - 1) / BM * a.ntn;
    DW_CHECK_CUDA(allow_smem(k64_gemm_tc<false>, smem64(kPl)));
    timer_begin("fp64_gemm", s);
    k64_gemm_tc<false><<<(unsigned)std::min<int64_t>(tiles, num_sms()), kThreads64, smem64(kPl), s>>>(ma, mb, a);
    timer_end("fp64_gemm", s, flops_of(rows, w), 0.0);
    count_launch();
    DW_CHECK_CUDA(launch_error());
    return DW_OK;
}

int gemm64_pipe(const double* A, int lda, const Weight64& w, double* C, int ldc, const Rows64& rows, int channels,
                const Epi64& e, cudaStream_t s) {
    Args64 a;
    a.A = A; a.lda = lda; a.W = w.w; a.ldw = w.ldw; a.C = C; a.ldc = ldc;
    a.ea = nullptr; a.ew = nullptr;
    a.rows = rows; a.e = e;
    a.N = w.N; a.K = w.K; a.channels = channels; a.ntn = 0;
    a.W64 = nullptr; a.per = 0; a.error = nullptr;
    int64_t most = 0;
    for (int g = 0; g < rows.ngroups; ++g) most = std::max(most, (int64_t)rows.B * rows.g[g].rpw);
    timer_begin("fp64_gemm", s);
    k64_gemm_pipe<<<dim3((w.N + 63) / 64, (unsigned)((most + 63) / 64), rows.ngroups), 256, 0, s>>>(a);
    timer_end("fp64_gemm", s, flops_of(rows, w), 0.0);
    count_launch();
    DW_CHECK_CUDA(launch_error());
    return DW_OK;
}

// Scratch of dets64_tangents for `m` matrices at a time.
struct DetScratch {
    Digits a, w;
    int* bal;
    double *E, *tr1, *tr2;
    size_t bytes;
};
static DetScratch carve_dets(int n, int T, int64_t m, void* base) {
    Carver c(base, (size_t)-1);
    DetScratch d;
    const int64_t per = (int64_t)(T - 1) * n;
    const int Kp = pad_k64(n);
    auto take = [&](int64_t rows) {
        __nv_bfloat16* dig = c.take<__nv_bfloat16>((size_t)planes64(true) * rows * Kp);
        return Digits{dig, c.take<int>(rows), rows, Kp, planes64(true)};
    };
    d.a = take(m * per);
    d.w = take(m * n);
    d.bal = c.take<int>(m * n);
    d.E = c.take<double>(m * per * n);
    d.tr1 = c.take<double>(m);
    d.tr2 = c.take<double>(m * (T - 1));
    d.bytes = c.used;
    return d;
}
// A matrix costs the FP64 loop (3 n + 1)(n^3 + n^2) FMAs and the digits (3 n + 1) n / 128 tiles whatever n:
// 4,096 matrices of 16 took 2.1 ms by the loop and 3.9 ms by digits, 376 of 27 1.6 and 1.2 ms, 1,536 of 40
// 29.9 and 12.8 ms (slicing, products and traces), so the line lies at 24. One tile holds up to 48 columns.
static bool dets64_fits(int n) { return n >= 24 && n <= BN; }

size_t dets64_scratch_bytes(int n, int T, int64_t nmat) {
    if (!dets64_fits(n) || T < 2) return 0;
    // up to 512 MB: some thousand tiles per launch
    const size_t one = carve_dets(n, T, 1, nullptr).bytes;
    const int64_t m = std::min<int64_t>(nmat, std::max<int64_t>(32, (int64_t)(((size_t)512 << 20) / one)));
    return carve_dets(n, T, m, nullptr).bytes + 256;
}

bool dets64_tangents(const double* MO64, const double* Ainv64, const double* sign, int n, int T, int K, int nmat,
                     const int* nvalid, int first, double* g, double* lapdet, void* scratch, size_t scratch_bytes, cudaStream_t s,
                     int* status) {
    *status = DW_OK;
    if (!dets64_fits(n) || T < 2 || !scratch) return false;
    char* base = reinterpret_cast<char*>(((uintptr_t)scratch + 255) / 256 * 256);
    const size_t lost = (size_t)(base - static_cast<char*>(scratch)), avail = scratch_bytes > lost ? scratch_bytes - lost : 0;
    int m = 0;                                       // the most matrices that the scratch holds
    for (int hi = nmat; m < hi;) {
        const int mid = m + (hi - m + 1) / 2;
        if (carve_dets(n, T, mid, nullptr).bytes <= avail) m = mid; else hi = mid - 1;
    }
    if (m < std::min(nmat, 32)) return false;
    const int per = (T - 1) * n;
    const DetScratch d = carve_dets(n, T, m, base);
    auto run = [&](int m0, int nm) -> int {
        Rows64 rows;                                 // the matrices' derivative channels: rows of n
        rows.ngroups = 1; rows.B = nm; rows.nvalid = nvalid; rows.mul = K; rows.first = first * K + m0;
        rows.g[0] = rows.g[1] = RowGroup{0, per, (int64_t)T * n, n};
        Rows64 cols = rows;                          // the inverses' columns
        cols.g[0] = cols.g[1] = RowGroup{0, n, (int64_t)n * n, 0};
        const double* A = MO64 + (int64_t)m0 * T * n * n;
        const double* W = Ainv64 + (int64_t)m0 * n * n;
        // The orbital index is balanced by powers of two, which leave the product as it is: an orbital that is
        // small at every electron has a large row of A^-1, and unscaled digits would lose the one's low bits
        // against the other orbitals (columns spread over 2^40: 2e-9 of the trace's terms, now 1e-18). The scale
        // comes from A^-1's rows: then a row of the product is off by n 2^-56 of its largest sum |dA| |A^-1| at
        // most, which scales by the columns of dA do not give.
        k64_balance<<<(unsigned)(((int64_t)nm * n + 7) / 8), 256, 0, s>>>(W, n, rows, d.bal);
        count_launch();
        k64_slice_rows<1, true><<<(unsigned)(((int64_t)nm * per + 7) / 8), 256, 0, s>>>(A, n, 1, n, rows, d.bal, 1, d.a);
        count_launch();
        k64_slice_rows<1, true><<<(unsigned)(((int64_t)nm * n + 7) / 8), 256, 0, s>>>(W, 1, n, n, cols, d.bal, -1, d.w);
        count_launch();
        CUtensorMap ma, mb;
        DW_CHECK(make_map3(&ma, d.a.dig, kDig, (int)d.a.rows, d.a.Kp, d.a.Kp, d.a.rows * d.a.Kp, BK, BM, kDig, false));
        DW_CHECK(make_map3(&mb, d.w.dig, kDig, (int)d.w.rows, d.w.Kp, d.w.Kp, d.w.rows * d.w.Kp, BK, BN, kDig, false));
        Args64 a;
        a.A = A; a.lda = n; a.W = nullptr; a.ldw = 0; a.C = d.E; a.ldc = n;
        a.ea = d.a.ex; a.ew = d.w.ex;
        a.rows = rows;
        a.N = n; a.K = n; a.channels = 1; a.ntn = 1;
        a.W64 = W; a.per = per;
        a.error = tc_error_flag();
        if (!a.error) return DW_ERR_CUDA;
        DW_CHECK_CUDA(allow_smem(k64_gemm_tc<true>, smem64(planes64(true))));
        const int64_t tiles = (int64_t)nm * ((per + BM - 1) / BM);
        k64_gemm_tc<true><<<(unsigned)std::min<int64_t>(tiles, num_sms()), kThreads64, smem64(planes64(true)), s>>>(ma, mb, a);
        count_launch();
        k64_traces<<<(unsigned)((int64_t)nm * (T - 1)), 128, (size_t)n * (n + 1) * sizeof(double), s>>>(
            d.E, sign + m0, n, T - 1, rows, g + (int64_t)m0 * (T - 2), d.tr1, d.tr2);
        count_launch();
        k64_lapdet<<<(nm + 7) / 8, 256, 0, s>>>(d.tr1, d.tr2, T - 1, rows, lapdet + m0);
        count_launch();
        DW_CHECK_CUDA(launch_error());
        return DW_OK;
    };
    for (int m0 = 0; m0 < nmat && *status == DW_OK; m0 += m) *status = run(m0, std::min(m, nmat - m0));
    return true;
}

}  // namespace dw

extern "C" {

// Test hook: C [M, N] = A [M, K] (row stride lda) @ W [K, N] (FP32, row stride ldw) by the digit products; ws
// holds the digit planes (dw_debug_gemm_fp64_bytes).
size_t dw_debug_gemm_fp64_bytes(int M, int N, int K) {
    return ((size_t)M + N) * dw::planes64(false) * dw::pad_k64(K) * 2 + ((size_t)M + N) * 4 + 4 * 256;
}
int dw_debug_gemm_fp64(const double* A, int lda, const float* W, int ldw, double* C, int M, int N, int K, void* ws,
                       void* stream) {
    using namespace dw;
    if (!tc_available()) return DW_ERR_UNSUPPORTED;
    if (!A || !W || !C || !ws || M <= 0 || N <= 0 || K <= 0 || K > kMaxK64) return DW_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    Carver c(ws, (size_t)-1);
    constexpr int kPl = planes64(false);
    Digits da{c.take<__nv_bfloat16>((size_t)kPl * M * pad_k64(K)), c.take<int>(M), M, pad_k64(K), kPl};
    Weight64 w{W, ldw, K, N, {c.take<__nv_bfloat16>((size_t)kPl * N * pad_k64(K)), c.take<int>(N), N, pad_k64(K), kPl}};
    const Rows64 rows = plain_rows(M, 1, nullptr);
    slice_rows64(A, lda, K, rows, da, s);
    slice_weights64(&w, 1, nullptr, s);
    return gemm64_tc(A, lda, da, w, C, N, rows, 1, Epi64(), s);
}

}  // extern "C"
