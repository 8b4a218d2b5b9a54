// FP64 form: the whole forward pass and the forward-Laplacian local energy in double precision
// (DW_PRECISION_FP64). It mirrors the reference's float64 mode (configuration.py:1893
// `float_precision`, applied through jax_enable_x64 in process_molecule.py:20-29): every GEMM,
// activation, convolution, envelope, LU, inverse, determinant tangent and reduction runs in FP64.
// The packed FP32 weights are read as they are (FP32 -> FP64 is exact), as the reference's x64
// mode evaluates float32-initialised weights in double.
//
// Layout. Every per-electron quantity carries C channels: C = 1 in value passes, C = 3n + 2 in
// tangent passes (channel 0 the value, 1 + 3m + c the derivative by coordinate c of electron m,
// C - 1 the Laplacian over all 3n coordinates). Rows are (walker, electron, channel); a linear map
// acts on every channel row alike (the bias only on channel 0) and an elementwise map couples the
// C rows of one (walker, electron). Pair streams depend on r only through d_ij and are carried as
// Taylor triples (f, df/dd, d2f/dd2); el-ion streams depend only on r_i and carry (value, three
// gradients, Laplacian) in r_i. This form is the precision anchor of the mixed form (and the FP64
// GPU rerun of its accuracy checks). The FP64 pipe of this part issues at a small fraction of the
// FP32 rate, so the GEMMs run as exact digit products on the tensor cores (fp64_gemm.cu).
#include "fp64_gemm.cuh"
#include <algorithm>

namespace dw {

// Launch family of one FP64 pass: dims, channel count, walkers in the chunk and an optional
// device-side count of valid walkers (walkers at or beyond it are skipped by every kernel).
struct Run64 {
    Dims d;
    int C;          // channels per electron
    int B;          // walkers in the chunk
    const int* nvalid;
    int first = 0;  // the chunk's first walker in that count
};
__device__ __forceinline__ int valid_walkers(const Run64& q) {
    return q.nvalid ? min(q.B, max(0, *q.nvalid - q.first)) : q.B;
}
__device__ __forceinline__ double softplus_d(double x) { return fmax(x, 0.0) + log1p(exp(-fabs(x))); }

// ------------------------------------------------------------------ elementwise tanh over channels
// Y = tanh(Z) for the C channel rows of each (walker, electron): value tanh(z0); gradient rows
// s z_t with s = 1 - tanh^2; Laplacian row s z_L - 2 tanh s sum_t z_t^2 (mlp.py:57-66 under the
// forward Laplacian).
__global__ void k64_jet_tanh(const double* __restrict__ Z, int ldz, int ncols, Run64 q, double* __restrict__ Y,
                             int ldy) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ent = idx / ncols;
    const int col = (int)(idx % ncols);
    if (ent >= (int64_t)valid_walkers(q) * q.d.n) return;
    const int C = q.C;
    const double* z = Z + ent * C * ldz + col;
    double* y = Y + ent * C * ldy + col;
    const double y0 = tanh(z[0]);
    y[0] = y0;
    if (C == 1) return;
    const double sp = 1.0 - y0 * y0;
    double sq = 0.0;
    for (int t = 1; t < C - 1; ++t) {
        const double zt = z[(int64_t)t * ldz];
        sq = fma(zt, zt, sq);
        y[(int64_t)t * ldy] = sp * zt;
    }
    y[(int64_t)(C - 1) * ldy] = sp * z[(int64_t)(C - 1) * ldz] - 2.0 * y0 * sp * sq;
}

static void jet_tanh(const double* Z, int ldz, int ncols, const Run64& q, double* Y, int ldy, cudaStream_t s) {
    const int64_t n = (int64_t)q.B * q.d.n * ncols;
    timer_begin("fp64_tanh", s);
    k64_jet_tanh<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(Z, ldz, ncols, q, Y, ldy);
    timer_end("fp64_tanh", s, 0.0, 0.0);
    count_launch();
}

// ------------------------------------------------------------------ ion maps
// him[seg][l][I][c] = tanh(ion_embed[Z_I - z_min] W_l + b_l)_c for c < eiw[l]
// (ferminet_embedding.py:171-175 h_ion_map, input_features.py:184-191 lookup); zero for Z = 0
// padding ions.
__global__ void k64_ion_maps(const float* __restrict__ P, ParamLayout L, Dims d, const int32_t* __restrict__ Zall,
                             double* __restrict__ him) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = d.nseg * 4 * d.N * 32;
    if (idx >= total) return;
    const int c = idx % 32, I = (idx / 32) % d.N, l = (idx / (32 * d.N)) % 4, g = idx / (32 * d.N * 4);
    const int z = Zall[g * d.N + I];
    double v = 0.0;
    if (z > 0 && c < d.eiw[l]) {
        const int zi = min(max(z - d.zmin, 0), d.zmax - d.zmin);
        const float* e = P + L.ion_embed + (int64_t)zi * d.EI;
        const float* w = P + L.h_ion_map_w[l];
        double acc = (double)P[L.h_ion_map_b[l] + c];
        for (int k = 0; k < d.EI; ++k) acc = fma((double)e[k], (double)w[k * d.eiw[l] + c], acc);
        v = tanh(acc);
    }
    him[idx] = v;
}

// ------------------------------------------------------------------ input features
// Layer-0 columns [d_iI, r_i - R_I] per ion, ion-major (input_features.py:41-68, :237-245), with
// their channels: gradients only along electron i's coordinates, Laplacian 2 / d for the distance.
__global__ void k64_features(const float* __restrict__ r, const float* __restrict__ Rall,
                             const int32_t* __restrict__ Zall, Run64 q, double* __restrict__ X, int ldx) {
    const Dims& d = q.d;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int I = (int)(idx % d.N);
    const int64_t row = idx / d.N;                 // (walker, electron, channel)
    const int t = (int)(row % q.C);
    const int64_t be = row / q.C;
    const int i = (int)(be % d.n);
    const int64_t b = be / d.n;
    if (b >= valid_walkers(q)) return;
    const int g = seg_of(d, b);
    const float* R = Rall + (int64_t)g * d.N * 3;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (Zall[g * d.N + I] > 0) {
        double df[3];
        for (int c = 0; c < 3; ++c) df[c] = (double)r[(b * d.n + i) * 3 + c] - (double)R[I * 3 + c];
        const double dist = sqrt(df[0] * df[0] + df[1] * df[1] + df[2] * df[2]);
        if (t == 0) {
            v[0] = dist; v[1] = df[0]; v[2] = df[1]; v[3] = df[2];
        } else if (t == q.C - 1) {
            v[0] = 2.0 / dist;
        } else if ((t - 1) / 3 == i) {
            const int c = (t - 1) % 3;
            v[0] = df[c] / dist;
            v[1 + c] = 1.0;
        }
    }
    double* o = X + row * ldx + I * 4;
    for (int k = 0; k < 4; ++k) o[k] = v[k];
}

// ------------------------------------------------------------------ pair streams (Taylor in d_ij)
// Warp per (walker, i, j), lane = feature column. Level-0 stream h = d_ij (zero with zero
// derivatives on the diagonal: get_distance_matrix pads the diagonal before the norm and zeroes
// it, utils/utils.py:287-305). Per level l: w = tanh(h W_w + b_w) with W_w = w_same / w_diff by
// the spins of i and j (ferminet_embedding.py:118-150); for l < 3 the stream update
// h <- residual(tanh(h W_h + b_h), h) (ferminet_embedding.py:246-262). Output
// WP[l][walker][i][j][{f, f', f''}][32].
__global__ void k64_pair_streams(const float* __restrict__ r, const float* __restrict__ P, ParamLayout L, Run64 q,
                                 double* __restrict__ WP) {
    const Dims& d = q.d;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int j = (int)(warp % d.n), i = (int)((warp / d.n) % d.n);
    const int64_t b = warp / ((int64_t)d.n * d.n);
    if (b >= valid_walkers(q)) return;
    const bool same = (i < d.nu) == (j < d.nu);
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;          // stream component held by this lane
    int width = 1;
    if (i != j && lane == 0) {
        const float* ri = r + (b * d.n + i) * 3;
        const float* rj = r + (b * d.n + j) * 3;
        double s = 0.0;
        for (int c = 0; c < 3; ++c) { const double x = (double)rj[c] - (double)ri[c]; s += x * x; }
        h0 = sqrt(s); h1 = 1.0; h2 = 0.0;
    }
    const int64_t plane = (int64_t)q.B * d.n * d.n * 96;
    for (int l = 0; l < 4; ++l) {
        for (int pass = 0; pass < (l < 3 ? 2 : 1); ++pass) {
            const int64_t wo = pass == 0 ? (same ? L.w_same_w[l] : L.w_diff_w[l]) : (same ? L.h_same_w[l] : L.h_diff_w[l]);
            const int64_t bo = pass == 0 ? (same ? L.w_same_b[l] : L.w_diff_b[l]) : (same ? L.h_same_b[l] : L.h_diff_b[l]);
            double z0 = (double)P[bo + lane], z1 = 0.0, z2 = 0.0;
            for (int k = 0; k < width; ++k) {
                const double x0 = __shfl_sync(0xffffffffu, h0, k), x1 = __shfl_sync(0xffffffffu, h1, k),
                             x2 = __shfl_sync(0xffffffffu, h2, k);
                const double w = (double)P[wo + k * 32 + lane];
                z0 = fma(x0, w, z0); z1 = fma(x1, w, z1); z2 = fma(x2, w, z2);
            }
            const double y0 = tanh(z0), sp = 1.0 - y0 * y0;
            const double y1 = sp * z1, y2 = sp * z2 - 2.0 * y0 * sp * z1 * z1;
            if (pass == 0) {
                double* o = WP + l * plane + (((b * d.n + i) * d.n + j) * 3) * 32 + lane;
                o[0] = y0; o[32] = y1; o[64] = y2;
            } else if (width == 32) {
                const double rs = 0.70710678118654752440;   // (old + new) / sqrt(2), mlp.py:13-17
                h0 = (h0 + y0) * rs; h1 = (h1 + y1) * rs; h2 = (h2 + y2) * rs;
            } else {
                h0 = y0; h1 = y1; h2 = y2;
            }
        }
        width = 32;
    }
}

// ------------------------------------------------------------------ el-ion streams
// Warp per (walker, electron), lane = feature column, loop over ions. Level-0 stream
// [d_iI, r_i - R_I] (width 4) with (value, three gradients, Laplacian) in r_i; per level the
// convolution conv_ei[i] = sum_I h_ei[i, I] * him[l][I] (ferminet_embedding.py:171-175) is
// accumulated, then for l < 3 h_ei <- residual(tanh(h_ei W + b), h_ei). Output
// CE[l][walker][i][5][32].
__global__ void k64_ei_streams(const float* __restrict__ r, const float* __restrict__ Rall,
                               const int32_t* __restrict__ Zall, const float* __restrict__ P, ParamLayout L,
                               const double* __restrict__ him, Run64 q, double* __restrict__ CE) {
    const Dims& d = q.d;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int i = (int)(warp % d.n);
    const int64_t b = warp / d.n;
    if (b >= valid_walkers(q)) return;
    const int g = seg_of(d, b);
    const float* R = Rall + (int64_t)g * d.N * 3;
    double acc[4][5];
    for (int l = 0; l < 4; ++l)
        for (int c = 0; c < 5; ++c) acc[l][c] = 0.0;
    for (int I = 0; I < d.N; ++I) {
        if (Zall[g * d.N + I] <= 0) continue;        // padding ion: contributes nothing
        double df[3];
        for (int c = 0; c < 3; ++c) df[c] = (double)r[(b * d.n + i) * 3 + c] - (double)R[I * 3 + c];
        const double dist = sqrt(df[0] * df[0] + df[1] * df[1] + df[2] * df[2]);
        double h[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (lane == 0) {
            h[0] = dist; h[1] = df[0] / dist; h[2] = df[1] / dist; h[3] = df[2] / dist; h[4] = 2.0 / dist;
        } else if (lane < 4) {
            h[0] = df[lane - 1]; h[lane] = 1.0;
        }
        int width = 4;
        for (int l = 0; l < 4; ++l) {
            const double hm = him[(((int64_t)g * 4 + l) * d.N + I) * 32 + lane];
            for (int c = 0; c < 5; ++c) acc[l][c] = fma(h[c], hm, acc[l][c]);
            if (l == 3) break;
            double z[5] = {(double)P[L.h_ei_b[l] + lane], 0.0, 0.0, 0.0, 0.0};
            for (int k = 0; k < width; ++k) {
                const double w = (double)P[L.h_ei_w[l] + k * 32 + lane];
                for (int c = 0; c < 5; ++c) z[c] = fma(__shfl_sync(0xffffffffu, h[c], k), w, z[c]);
            }
            const double y0 = tanh(z[0]), sp = 1.0 - y0 * y0;
            double y[5];
            y[0] = y0;
            y[1] = sp * z[1]; y[2] = sp * z[2]; y[3] = sp * z[3];
            y[4] = sp * z[4] - 2.0 * y0 * sp * (z[1] * z[1] + z[2] * z[2] + z[3] * z[3]);
            const double rs = width == 32 ? 0.70710678118654752440 : 1.0;
            for (int c = 0; c < 5; ++c) h[c] = width == 32 ? (h[c] + y[c]) * rs : y[c];
            width = 32;
        }
    }
    const int64_t plane = (int64_t)q.B * d.n * 5 * 32;
    for (int l = 0; l < 4; ++l)
        for (int c = 0; c < 5; ++c) CE[l * plane + ((b * d.n + i) * 5 + c) * 32 + lane] = acc[l][c];
}

// ------------------------------------------------------------------ SchNet el-el convolution
// conv_ee[i] = sum_j w_ij * h_map_j (ferminet_embedding.py:152-169, self-pair included) with the
// product rule over the channels: w_ij depends on r only through d_ij (gradient u = (r_i - r_j) /
// d_ij along r_i, -u along r_j; |grad d|^2 = 2, Lap d = 4 / d). Thread per (channel, column) of one
// (walker, electron) block; writes columns [col0, col0 + 32) of the layer input. Columns [col0 + 32,
// col0 + 32 + eiw) take conv_ei of the level: value, electron i's own gradient rows and the
// Laplacian, zero elsewhere.
__global__ void k64_conv(const float* __restrict__ r, const double* __restrict__ WPl, const double* __restrict__ HM,
                         const double* __restrict__ CEl, int eiw, Run64 q, double* __restrict__ X, int ldx, int col0) {
    const Dims& d = q.d;
    const int i = blockIdx.x % d.n;
    const int64_t b = blockIdx.x / d.n;
    if (b >= valid_walkers(q)) return;
    const int C = q.C, n = d.n;
    __shared__ double u_sh[kMaxEl][4];       // u_ij (3) and 1 / d_ij
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        double df[3], s = 0.0;
        for (int c = 0; c < 3; ++c) {
            df[c] = (double)r[(b * n + i) * 3 + c] - (double)r[(b * n + j) * 3 + c];
            s += df[c] * df[c];
        }
        const double dist = sqrt(s);
        const double inv = j == i ? 0.0 : 1.0 / dist;
        for (int c = 0; c < 3; ++c) u_sh[j][c] = df[c] * inv;
        u_sh[j][3] = inv;
    }
    __syncthreads();
    const double* wp = WPl + ((b * n + i) * n) * 96;      // [j][3][32]
    const double* hm = HM + (b * n) * C * 32;             // [(j, t)][32]
    for (int e = threadIdx.x; e < C * 32; e += blockDim.x) {
        const int t = e / 32, col = e % 32;
        double v = 0.0;
        for (int j = 0; j < n; ++j) v = fma(wp[j * 96 + col], hm[((int64_t)j * C + t) * 32 + col], v);
        if (t > 0 && t < C - 1) {
            const int m = (t - 1) / 3, c = (t - 1) % 3;
            if (m == i) {
                for (int j = 0; j < n; ++j) {
                    if (j == i) continue;
                    v = fma(wp[j * 96 + 32 + col] * u_sh[j][c], hm[((int64_t)j * C) * 32 + col], v);
                }
            } else {
                v = fma(-wp[m * 96 + 32 + col] * u_sh[m][c], hm[((int64_t)m * C) * 32 + col], v);
            }
        } else if (t == C - 1 && C > 1) {
            for (int j = 0; j < n; ++j) {
                if (j == i) continue;
                const double w1 = wp[j * 96 + 32 + col], w2 = wp[j * 96 + 64 + col];
                const double lapw = 2.0 * w2 + 4.0 * w1 * u_sh[j][3];
                double cross = 0.0;
                for (int c = 0; c < 3; ++c)
                    cross = fma(u_sh[j][c], hm[((int64_t)j * C + 1 + 3 * i + c) * 32 + col] -
                                             hm[((int64_t)j * C + 1 + 3 * j + c) * 32 + col], cross);
                v = fma(lapw, hm[((int64_t)j * C) * 32 + col], v);
                v = fma(2.0 * w1, cross, v);
            }
        }
        X[(((b * n + i) * C) + t) * (int64_t)ldx + col0 + col] = v;
    }
    const double* ce = CEl + (b * n + i) * 5 * 32;
    for (int e = threadIdx.x; e < C * eiw; e += blockDim.x) {
        const int t = e / eiw, col = e % eiw;
        double v = 0.0;
        if (t == 0) v = ce[col];
        else if (t == C - 1) v = ce[4 * 32 + col];
        else if ((t - 1) / 3 == i) v = ce[(1 + (t - 1) % 3) * 32 + col];
        X[(((b * n + i) * C) + t) * (int64_t)ldx + col0 + 32 + col] = v;
    }
}

// ------------------------------------------------------------------ envelope orbitals
// MO[b][k][t][i][o] = env_i(k, o) * BF[(b, i, t)][k n + o] with the product rule; the isotropic
// exponential envelope env = sum_I w exp(-softplus(alpha) d_iI) (envelope_orbitals.py:96-127)
// depends only on r_i: gradient -a e u, Laplacian e (a^2 - 2 a / d).
__global__ void k64_envelope_mo(const float* __restrict__ r, const float* __restrict__ Rall,
                                const int32_t* __restrict__ Zall, const float* __restrict__ P, ParamLayout L, Run64 q,
                                const double* __restrict__ BF, int ldbf, double* __restrict__ MO) {
    const Dims& d = q.d;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int n = d.n, C = q.C;
    const int o = (int)(idx % n);
    const int i = (int)((idx / n) % n);
    const int k = (int)((idx / ((int64_t)n * n)) % d.K);
    const int64_t b = idx / ((int64_t)n * n * d.K);
    if (b >= valid_walkers(q)) return;
    const int g = seg_of(d, b);
    const float* R = Rall + (int64_t)g * d.N * 3;
    const bool up = i < d.nu;
    const int64_t col = (int64_t)k * n + o;
    const float* alpha = P + (up ? L.alpha_up : L.alpha_dn);
    const float* wts = P + (up ? L.weights_up : L.weights_dn);
    double e0 = 0.0, eg[3] = {0.0, 0.0, 0.0}, eL = 0.0;
    for (int I = 0; I < d.N; ++I) {
        if (Zall[g * d.N + I] <= 0) continue;
        double df[3];
        for (int c = 0; c < 3; ++c) df[c] = (double)r[(b * n + i) * 3 + c] - (double)R[I * 3 + c];
        const double dist = sqrt(df[0] * df[0] + df[1] * df[1] + df[2] * df[2]);
        const double a = softplus_d((double)alpha[(int64_t)I * d.KN + col]);
        const double e = (double)wts[(int64_t)I * d.KN + col] * exp(-a * dist);
        e0 += e;
        if (C > 1) {
            for (int c = 0; c < 3; ++c) eg[c] -= a * e * df[c] / dist;
            eL += e * (a * a - 2.0 * a / dist);
        }
    }
    const double* bf = BF + ((b * n + i) * C) * (int64_t)ldbf + col;
    double* mo = MO + (((b * d.K + k) * C) * n + i) * (int64_t)n + o;
    const int64_t plane = (int64_t)n * n;
    const double b0 = bf[0];
    mo[0] = e0 * b0;
    if (C == 1) return;
    for (int t = 1; t < C - 1; ++t) {
        double v = e0 * bf[(int64_t)t * ldbf];
        if ((t - 1) / 3 == i) v = fma(eg[(t - 1) % 3], b0, v);
        mo[t * plane] = v;
    }
    double lap = fma(eL, b0, e0 * bf[(int64_t)(C - 1) * ldbf]);
    for (int c = 0; c < 3; ++c) lap = fma(2.0 * eg[c], bf[(int64_t)(1 + 3 * i + c) * ldbf], lap);
    mo[(C - 1) * plane] = lap;
}

// ------------------------------------------------------------------ determinants
// FP64 Gauss-Jordan elimination with partial pivoting of the value-channel Slater matrix of one
// (walker, determinant): log|det|, sign (jnp.linalg.slogdet, wavefunction.py:69-73) and, in
// tangent passes, the inverse. Block of 128 threads, [A | I] in shared memory.
__global__ void __launch_bounds__(128)
k64_slogdet_inv(const double* __restrict__ MO, Run64 q, double* __restrict__ logdet, double* __restrict__ sign,
                double* __restrict__ Ainv) {
    const Dims& d = q.d;
    const int n = d.n, C = q.C, w2 = 2 * n + 1;
    const int64_t mat = blockIdx.x;                  // b * K + k
    if (mat / d.K >= valid_walkers(q)) return;
    extern __shared__ double aug[];                  // [n][2n + 1], then n factors
    double* fac = aug + (int64_t)n * w2;
    __shared__ int s_piv;
    __shared__ double s_pv, s_logabs, s_sign;
    const int tid = threadIdx.x;
    const double* A = MO + (mat * C) * (int64_t)n * n;
    const bool want_inv = Ainv != nullptr;
    const int cols = want_inv ? 2 * n : n;
    for (int e = tid; e < n * 2 * n; e += blockDim.x) {
        const int rr = e / (2 * n), cc = e % (2 * n);
        aug[rr * w2 + cc] = cc < n ? A[rr * n + cc] : (cc - n == rr ? 1.0 : 0.0);
    }
    if (tid == 0) { s_logabs = 0.0; s_sign = 1.0; }
    __syncthreads();
    bool singular = false;
    for (int p = 0; p < n; ++p) {
        if (tid < 32) {
            double best = -1.0; int bi = p;
            for (int rr = p + tid; rr < n; rr += 32) {
                const double v = fabs(aug[rr * w2 + p]);
                if (v > best) { best = v; bi = rr; }
            }
            for (int off = 16; off > 0; off >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, best, off);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            // the pivot itself is handed over too: a warp that read it from the matrix could come after the
            // first warp has exchanged the rows
            if (tid == 0) { s_piv = bi; s_pv = aug[bi * w2 + p]; }
        }
        __syncthreads();
        const int piv = s_piv;
        const double pv = s_pv;
        if (pv == 0.0 || !isfinite(pv)) { singular = true; break; }
        if (piv != p) {
            for (int cc = p + tid; cc < cols; cc += blockDim.x) {
                const double x = aug[p * w2 + cc];
                aug[p * w2 + cc] = aug[piv * w2 + cc];
                aug[piv * w2 + cc] = x;
            }
        }
        __syncthreads();
        const double inv = 1.0 / pv;
        if (tid == 0) {
            s_logabs += log(fabs(pv));
            s_sign *= (pv < 0.0) != (piv != p) ? -1.0 : 1.0;
        }
        for (int cc = p + 1 + tid; cc < cols; cc += blockDim.x) aug[p * w2 + cc] *= inv;
        for (int rr = tid; rr < n; rr += blockDim.x) fac[rr] = aug[rr * w2 + p];
        __syncthreads();
        const int span = cols - (p + 1);
        for (int e = tid; e < n * span; e += blockDim.x) {
            const int rr = e / span, cc = p + 1 + e % span;
            if (rr == p || (!want_inv && rr < p)) continue;   // value passes: LU rows only
            aug[rr * w2 + cc] = fma(-fac[rr], aug[p * w2 + cc], aug[rr * w2 + cc]);
        }
        __syncthreads();
    }
    if (tid == 0) {
        logdet[mat] = singular ? -INFINITY : s_logabs;
        sign[mat] = singular ? 0.0 : s_sign;
    }
    if (want_inv) {
        double* out = Ainv + mat * (int64_t)n * n;
        for (int e = tid; e < n * n; e += blockDim.x) out[e] = singular ? 0.0 : aug[(e / n) * w2 + n + e % n];
    }
}

// g_t = tr(A^-1 dA_t) over the 3n gradient channels and lap = tr(A^-1 Lap A) - sum_t tr((A^-1 dA_t)^2)
// of one (walker, determinant), all in FP64.
__global__ void __launch_bounds__(128)
k64_det_tangents(const double* __restrict__ MO, const double* __restrict__ Ainv, const double* __restrict__ sign,
                 Run64 q, double* __restrict__ g, double* __restrict__ lapdet) {
    const Dims& d = q.d;
    const int n = d.n, C = q.C, n3 = 3 * n, nn = n * n;
    const int64_t mat = blockIdx.x;
    if (mat / d.K >= valid_walkers(q)) return;
    extern __shared__ double sm[];
    double* Ai = sm;
    double* dA = Ai + nn;
    double* Cm = dA + nn;
    __shared__ double red[2][4];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (sign[mat] == 0.0) {
        for (int t = tid; t < n3; t += blockDim.x) g[mat * n3 + t] = 0.0;
        if (tid == 0) lapdet[mat] = 0.0;
        return;
    }
    for (int e = tid; e < nn; e += blockDim.x) Ai[e] = Ainv[mat * nn + e];
    double lap_acc = 0.0;
    for (int t = 1; t < C; ++t) {
        const double* src = MO + ((mat * C) + t) * (int64_t)nn;
        __syncthreads();
        for (int e = tid; e < nn; e += blockDim.x) dA[e] = src[e];
        __syncthreads();
        double tr = 0.0, tr2 = 0.0;
        for (int e = tid; e < nn; e += blockDim.x) {
            const int a = e / n, c = e % n;
            double acc = 0.0;
            for (int m = 0; m < n; ++m) acc = fma(Ai[a * n + m], dA[m * n + c], acc);
            Cm[e] = acc;
            if (a == c) tr += acc;
        }
        __syncthreads();
        if (t != C - 1)
            for (int e = tid; e < nn; e += blockDim.x) tr2 = fma(Cm[e], Cm[(e % n) * n + e / n], tr2);
        tr = warp_sum(tr); tr2 = warp_sum(tr2);
        if (lane == 0) { red[0][wid] = tr; red[1][wid] = tr2; }
        __syncthreads();
        if (tid == 0) {
            const double s0 = red[0][0] + red[0][1] + red[0][2] + red[0][3];
            const double s1 = red[1][0] + red[1][1] + red[1][2] + red[1][3];
            if (t == C - 1) lap_acc += s0;
            else { g[mat * n3 + (t - 1)] = s0; lap_acc -= s1; }
        }
    }
    if (tid == 0) lapdet[mat] = lap_acc;
}

// By digit products where they are faster and the scratch holds enough matrices, else by k64_det_tangents.
static int launch_tangents64(const double* MO, const double* Ainv, const double* sign, const Run64& q, int nmat, double* g,
                             double* lapdet, void* scratch, size_t scratch_bytes, cudaStream_t s) {
    const int n = q.d.n;
    int status = DW_OK;
    if (dets64_tangents(MO, Ainv, sign, n, q.C, q.d.K, nmat, q.nvalid, q.first, g, lapdet, scratch, scratch_bytes, s, &status)) return status;
    const size_t sm = (size_t)3 * n * n * sizeof(double);
    if (sm > 48 * 1024) allow_smem(k64_det_tangents, 3 * kMaxEl * kMaxEl * (int)sizeof(double));
    k64_det_tangents<<<nmat, 128, sm, s>>>(MO, Ainv, sign, q, g, lapdet);
    count_launch();
    return DW_OK;
}

// Jastrow output: jas[(b, t)] = sum_i sum_c J2[(b, i, t)][c] w2[c] (wavefunction.py:57-59, linear
// output without bias, summed over electrons). Warp per (walker, channel).
__global__ void k64_jastrow_out(const double* __restrict__ J2, int ldj, const float* __restrict__ w2, Run64 q,
                                double* __restrict__ jas) {
    const Dims& d = q.d;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int t = (int)(warp % q.C);
    const int64_t b = warp / q.C;
    if (b >= valid_walkers(q)) return;
    double acc = 0.0;
    for (int i = 0; i < d.n; ++i) {
        const double* row = J2 + ((b * d.n + i) * q.C + t) * (int64_t)ldj;
        for (int c = lane; c < d.J1; c += 32) acc = fma(row[c], (double)w2[c], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) jas[b * q.C + t] = acc;
}

// ------------------------------------------------------------------ plan and launch sequence
struct Plan64 {
    int Bc, C;
    double* him;
    double *XA, *XB, *Zt, *HM, *M, *WB, *WP, *CE, *BF, *MO, *logdet, *sign, *Ainv, *g, *lapdet, *J1, *J2, *jas;
    void* scratch; size_t scratch_bytes;             // dets64_tangents
    Digits act, mean;              // digit planes of the activation rows and of the spin-mean rows
    Weight64 w[kMaxW64];           // h_map[4], mean rows[4], main rows[4], backflow[2], Jastrow[2] (w.w set per call)
    size_t bytes;
};
static const int kXW64 = 320;    // layer 1..3 input [h (256) | conv_ee (32) | conv_ei (32)]

// Buffers of a chunk of Bc walkers, with the digit planes and the tangents' scratch or without.
static Plan64 carve64(const Dims& d, int C, int Bc, void* ws, bool digits = true) {
    Carver c(ws, (size_t)-1);
    Plan64 p;
    p.Bc = Bc; p.C = C;
    const int64_t rows = (int64_t)Bc * d.n * C;
    const int w0 = d.hw[0] + d.E + d.eiw[0];
    p.him = c.take<double>((size_t)kMaxSeg * 4 * d.N * 32);
    p.XA = c.take<double>(rows * kXW64);
    p.XB = c.take<double>(rows * std::max(kXW64, w0));
    p.Zt = c.take<double>(rows * std::max(d.D, d.J0));
    p.HM = c.take<double>(rows * 32);
    p.M = c.take<double>((int64_t)Bc * C * 2 * d.D);
    p.WB = c.take<double>((int64_t)Bc * C * d.D);
    p.WP = c.take<double>((int64_t)4 * Bc * d.n * d.n * 96);
    p.CE = c.take<double>((int64_t)4 * Bc * d.n * 5 * 32);
    p.BF = c.take<double>(rows * d.KN);
    p.MO = c.take<double>((int64_t)Bc * d.K * C * d.n * d.n);
    p.logdet = c.take<double>((int64_t)Bc * d.K);
    p.sign = c.take<double>((int64_t)Bc * d.K);
    if (C > 1) {
        p.Ainv = c.take<double>((int64_t)Bc * d.K * d.n * d.n);
        p.g = c.take<double>((int64_t)Bc * d.K * 3 * d.n);
        p.lapdet = c.take<double>((int64_t)Bc * d.K);
    } else {
        p.Ainv = p.g = p.lapdet = nullptr;
    }
    p.J1 = c.take<double>(rows * d.J0);
    p.J2 = c.take<double>(rows * d.J1);
    p.jas = c.take<double>((int64_t)Bc * C);
    p.scratch = nullptr;
    p.scratch_bytes = 0;
    if (digits && C > 1) {
        p.scratch_bytes = dets64_scratch_bytes(d.n, C, (int64_t)Bc * d.K);
        p.scratch = c.take<unsigned char>(p.scratch_bytes);
    }
    auto take = [&](int64_t r, int K) {
        const int Kp = pad_k64(K);
        if (!digits) return Digits{nullptr, nullptr, r, Kp, 0};
        __nv_bfloat16* dig = c.take<__nv_bfloat16>((size_t)planes64(false) * r * Kp);
        return Digits{dig, c.take<int>(r), r, Kp, planes64(false)};
    };
    p.act = take(rows, std::max(kXW64, w0));
    p.mean = take((int64_t)Bc * C, 2 * std::max(d.D, d.hw[0]));
    const int J[2] = {d.J0, d.J1}, JK[2] = {d.D, d.J0};
    for (int k = 0; k < kMaxW64; ++k) {
        const int l = k % 4;
        const int K = k < 4 ? d.hw[l] : k < 8 ? 2 * d.hw[l] : k < 12 ? d.hw[l] + d.E + d.eiw[l] : k < 14 ? d.D : JK[k - 14];
        const int N = k < 4 ? d.E : k < 12 ? d.D : k < 14 ? d.KN : J[k - 14];
        p.w[k] = Weight64{nullptr, N, K, N, take(N, K)};
    }
    p.bytes = c.used;
    return p;
}

static const size_t kChunkBudget64 = (size_t)6 << 30;

// Walkers of a chunk with the digit planes: the most whose buffers take `budget` bytes (0: not one).
static int choose_chunk64_digits(const Dims& d, int C, int B, size_t budget) {
    int lo = 0;
    for (int hi = std::min(B, 32768); lo < hi;) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (carve64(d, C, mid, nullptr).bytes <= budget) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// Walkers of a chunk without them.
static int choose_chunk64(const Dims& d, int C, int B, size_t budget) {
    const size_t one = carve64(d, C, 1, nullptr, false).bytes, two = carve64(d, C, 2, nullptr, false).bytes;
    const size_t per = std::max<size_t>(two > one ? two - one : one, 1);
    const size_t fixed = one > per ? one - per : 0;
    const size_t avail = budget > fixed ? budget - fixed : per;
    int bc = std::min((int)std::min<size_t>(std::max<size_t>(1, avail / per), 32768), B);
    while (bc > 1 && carve64(d, C, bc, nullptr, false).bytes > budget) bc -= std::max(1, bc / 32);
    return bc;
}

static inline unsigned blocks_for(int64_t n, int tpb) { return (unsigned)((n + tpb - 1) / tpb); }

// The FP64 forward (value or tangent) of one chunk of walkers.
static int run_chunk64(const Plan64& p, const Dims& d0, int Bc, const float* P, const ParamLayout& L, const float* r,
                       const float* R, const int32_t* Z, const int32_t* seg, const int* nvalid, int first, float* lp,
                       float* phase, float* E, float* grad, cudaStream_t s) {
    Dims d = d0;
    d.seg = seg;
    Run64 q;
    q.d = d; q.C = p.C; q.B = Bc; q.nvalid = nvalid; q.first = first;
    const int C = p.C, n = d.n;
    const bool digits = p.act.dig != nullptr;
    const int64_t rows = (int64_t)Bc * n * C;
    const bool tang = C > 1;
    const int w0 = d.hw[0] + d.E + d.eiw[0];
    Rows64 all = plain_rows(Bc, n * C, nvalid), chan = plain_rows(Bc, C, nvalid);
    all.first = chan.first = first;
    // digit planes of the first K columns, reusing the plan's buffer at that width
    auto planes = [](Digits x, int K) { x.Kp = pad_k64(K); return x; };
    auto slice = [&](const double* A, int lda, int K, const Rows64& rr) {
        const Digits x = planes(p.act, K);
        if (digits) slice_rows64(A, lda, K, rr, x, s);
        return x;
    };
    auto gemm = [&](const double* A, int lda, const Digits& da, const Weight64& w, double* Cm, int ldc, const Rows64& rr,
                    const Epi64& e) {
        return digits ? gemm64_tc(A, lda, da, w, Cm, ldc, rr, C, e, s) : gemm64_pipe(A, lda, w, Cm, ldc, rr, C, e, s);
    };
    // layer-0 input [features | conv_ee | conv_ei] in XB (free until layer 1 writes it)
    timer_begin("fp64_streams", s);
    k64_features<<<blocks_for(rows * d.N, 256), 256, 0, s>>>(r, R, Z, q, p.XB, w0);
    count_launch();
    k64_pair_streams<<<blocks_for((int64_t)Bc * n * n * 32, 256), 256, 0, s>>>(r, P, L, q, p.WP);
    count_launch();
    k64_ei_streams<<<blocks_for((int64_t)Bc * n * 32, 256), 256, 0, s>>>(r, R, Z, P, L, p.him, q, p.CE);
    count_launch();
    timer_end("fp64_streams", s, 0.0, 0.0);
    double* xin = p.XB;
    int ldin = w0;
    for (int l = 0; l < 4; ++l) {
        double* xout = (l % 2 == 0) ? p.XA : p.XB;
        const int hw = d.hw[l];
        // h_map = tanh(h W + b) -> HM
        Epi64 em; em.bias = P + L.h_map_b[l];
        const Digits dh = slice(xin, ldin, hw, all);
        DW_CHECK(gemm(xin, ldin, dh, p.w[l], p.Zt, d.E, all, em));
        jet_tanh(p.Zt, d.E, d.E, q, p.HM, 32, s);
        // convolutions into columns [hw, hw + E + eiw)
        timer_begin("fp64_conv", s);
        k64_conv<<<(unsigned)((int64_t)Bc * n), 128, 0, s>>>(r, p.WP + (int64_t)l * Bc * n * n * 96, p.HM,
                                                              p.CE + (int64_t)l * Bc * n * 5 * 32, d.eiw[l], q, xin, ldin,
                                                              hw);
        timer_end("fp64_conv", s, 0.0, 0.0);
        count_launch();
        // spin means and their per-(walker, channel) product with the mean rows (+ the layer bias)
        const Digits dm = planes(p.mean, 2 * hw);
        spin_means64(xin, ldin, hw, n, d.nu, C, chan, p.M, dm, s);
        Epi64 eb; eb.bias = P + L.h_el_b[l];
        DW_CHECK(gemm(p.M, 2 * hw, dm, p.w[4 + l], p.WB, d.D, chan, eb));
        // h_el = tanh([h | conv_ee | conv_ei] W_main + mean term) (ferminet_embedding.py:233-241)
        Epi64 e3; e3.rowbias = p.WB; e3.ldrb = d.D;
        const Digits dx = slice(xin, ldin, p.w[8 + l].K, all);
        DW_CHECK(gemm(xin, ldin, dx, p.w[8 + l], p.Zt, d.D, all, e3));
        jet_tanh(p.Zt, d.D, d.D, q, xout, kXW64, s);
        xin = xout;
        ldin = kXW64;
    }
    const double* H = xin;
    // The final embedding's digit rows ordered by spin, then walker: backflow of each spin's rows
    // (envelope_orbitals.py:46-75), and the Jastrow layer over both groups.
    Rows64 spins = all;
    spins.ngroups = 2;
    spins.g[0] = RowGroup{0, d.nu * C, (int64_t)n * C, 0};
    spins.g[1] = RowGroup{(int64_t)Bc * d.nu * C, d.nd * C, (int64_t)n * C, (int64_t)d.nu * C};
    const Digits dH = slice(H, kXW64, d.D, spins);
    for (int spin = 0; spin < 2; ++spin) {
        Rows64 one = spins;
        one.ngroups = 1;
        one.g[0] = spins.g[spin];
        DW_CHECK(gemm(H, kXW64, dH, p.w[12 + spin], p.BF, d.KN, one, Epi64()));
    }
    timer_begin("fp64_envelope", s);
    k64_envelope_mo<<<blocks_for((int64_t)Bc * d.K * n * n, 128), 128, 0, s>>>(r, R, Z, P, L, q, p.BF, d.KN, p.MO);
    timer_end("fp64_envelope", s, 0.0, 0.0);
    count_launch();
    const int nmat = Bc * d.K;
    const size_t sm_lu = ((size_t)n * (2 * n + 1) + n) * sizeof(double);
    if (sm_lu > 48 * 1024) allow_smem(k64_slogdet_inv, (kMaxEl * (2 * kMaxEl + 1) + kMaxEl) * (int)sizeof(double));
    timer_begin("fp64_lu", s);
    k64_slogdet_inv<<<nmat, 128, sm_lu, s>>>(p.MO, q, p.logdet, p.sign, tang ? p.Ainv : nullptr);
    timer_end("fp64_lu", s, 0.0, 0.0);
    count_launch();
    if (tang) {
        timer_begin("fp64_det_tangents", s);
        DW_CHECK(launch_tangents64(p.MO, p.Ainv, p.sign, q, nmat, p.g, p.lapdet, p.scratch, p.scratch_bytes, s));
        timer_end("fp64_det_tangents", s, 0.0, 0.0);
    }
    // Jastrow MLP([64, 64, 1]) on the final embedding (wavefunction.py:42-60)
    Epi64 j0; j0.bias = P + L.jas_b[0];
    DW_CHECK(gemm(H, kXW64, dH, p.w[14], p.Zt, d.J0, spins, j0));
    jet_tanh(p.Zt, d.J0, d.J0, q, p.J1, d.J0, s);
    Epi64 j1; j1.bias = P + L.jas_b[1];
    const Digits dj = slice(p.J1, d.J0, d.J0, all);
    DW_CHECK(gemm(p.J1, d.J0, dj, p.w[15], p.Zt, d.J1, all, j1));
    jet_tanh(p.Zt, d.J1, d.J1, q, p.J2, d.J1, s);
    k64_jastrow_out<<<blocks_for((int64_t)Bc * C * 32, 256), 256, 0, s>>>(p.J2, d.J1, P + L.jas_w[2], q, p.jas);
    count_launch();
    // log-sum-exp over determinants, derivatives of log psi^2, kinetic + FP64 Coulomb energy
    Dims dc = d;
    dc.Tp = C;
    launch_combine(p.logdet, p.sign, p.g, p.lapdet, p.jas, r, R, Z, dc, Bc, lp, phase, E, grad, s, 1, nvalid, nullptr, first);
    DW_CHECK_CUDA(launch_error());
    return DW_OK;
}

// FP64 determinant algebra on float32 Slater-matrix channels MO[b][k][t][i][o] (t < d.T): the
// channels are widened to FP64 in MO64, then the FP64 LU / Gauss-Jordan inverse and the FP64
// determinant tangents of this file give log|det|, sign, the gradient traces and the Laplacian
// term. Used by the plain form's FP64-determinant variant.
__global__ void k64_widen(const float* __restrict__ x, int64_t n, double* __restrict__ y) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = (double)x[i];
}

int fp64_dets_from_f32(const float* MO, const Dims& d, int Bc, double* MO64, double* Ainv64, double* logdet,
                       double* sign, double* g, double* lapdet, void* scratch, size_t scratch_bytes, cudaStream_t s) {
    Run64 q;
    q.d = d; q.C = d.T; q.B = Bc; q.nvalid = nullptr;
    const int n = d.n, nmat = Bc * d.K;
    const int64_t ne = (int64_t)nmat * d.T * n * n;
    k64_widen<<<(unsigned)std::min<int64_t>((ne + 255) / 256, 152 * 32), 256, 0, s>>>(MO, ne, MO64);
    count_launch();
    const bool tang = d.T > 1;
    const size_t sm_lu = ((size_t)n * (2 * n + 1) + n) * sizeof(double);
    if (sm_lu > 48 * 1024) allow_smem(k64_slogdet_inv, (kMaxEl * (2 * kMaxEl + 1) + kMaxEl) * (int)sizeof(double));
    k64_slogdet_inv<<<nmat, 128, sm_lu, s>>>(MO64, q, logdet, sign, tang ? Ainv64 : nullptr);
    count_launch();
    if (tang) DW_CHECK(launch_tangents64(MO64, Ainv64, sign, q, nmat, g, lapdet, scratch, scratch_bytes, s));
    DW_CHECK_CUDA(launch_error());
    return DW_OK;
}

int fp64_max_chunk(const DwArch* a, bool tang) {
    Dims d = make_dims(a, tang);
    const int C = tang ? 3 * d.n + 2 : 1;
    return choose_chunk64(d, C, 1 << 30, kChunkBudget64);
}

size_t fp64_least_bytes(const DwArch* a, int B, bool tang) {
    Dims d = make_dims(a, tang);
    const int C = tang ? 3 * d.n + 2 : 1;
    return (carve64(d, C, choose_chunk64(d, C, std::max(B, 1), kChunkBudget64), nullptr, false).bytes + 4096 + 255) / 256 * 256;
}
size_t fp64_plan_bytes(const DwArch* a, int B, bool tang) {
    Dims d = make_dims(a, tang);
    const int C = tang ? 3 * d.n + 2 : 1;
    const int bc = std::max(1, choose_chunk64_digits(d, C, std::max(B, 1), kChunkBudget64));
    return std::max((carve64(d, C, bc, nullptr).bytes + 4096 + 255) / 256 * 256, fp64_least_bytes(a, B, tang));
}

int fp64_forward_all(const DwArch* a, const float* P, const void* prepared, const float* r, int B, const float* R,
                     const int32_t* Z, float* lp, float* phase, float* E, float* grad, bool tang, void* ws,
                     size_t ws_bytes, cudaStream_t s, const int32_t* seg, int nseg, const int* nvalid) {
    Dims d = make_dims(a, tang);
    if (nseg < 1 || nseg > kMaxSeg || (nseg > 1 && !seg)) return DW_ERR_ARG;
    const int C = tang ? 3 * d.n + 2 : 1;
    d.T = C; d.Tp = C; d.lap = tang ? C - 1 : -1;
    d.nseg = nseg;
    ParamLayout L;
    make_layout(a, &L);
    const float* main_w[4];
    const float* mean_w[4];
    prepared_fp32_layers(a, prepared, main_w, mean_w);
    // With the digit planes in the largest chunk that the region holds (its base rounded up to 256 bytes: the
    // planes are read by TMA), or, in a region sized without them that holds not one walker's, without.
    int bc = choose_chunk64(d, C, B, kChunkBudget64);
    if (carve64(d, C, bc, nullptr, false).bytes > ws_bytes) return DW_ERR_WORKSPACE;
    char* base = reinterpret_cast<char*>(((uintptr_t)ws + 255) / 256 * 256);
    const size_t lost = (size_t)(base - static_cast<char*>(ws)), room = ws_bytes > lost ? ws_bytes - lost : 0;
    const size_t one = carve64(d, C, 1, nullptr).bytes;      // one walker may take more than the budget
    const int bd = one > room ? 0 : std::max(1, choose_chunk64_digits(d, C, B, std::min(room, kChunkBudget64)));
    if (bd > 0) bc = bd;
    Plan64 p = bd > 0 ? carve64(d, C, bc, base) : carve64(d, C, bc, ws, false);
    for (int l = 0; l < 4; ++l) {
        p.w[l].w = P + L.h_map_w[l];
        p.w[4 + l].w = mean_w[l];
        p.w[8 + l].w = main_w[l];
    }
    p.w[12].w = P + L.bf_up;
    p.w[13].w = P + L.bf_dn;
    p.w[14].w = P + L.jas_w[0];
    p.w[15].w = P + L.jas_w[1];
    if (p.act.dig) slice_weights64(p.w, kMaxW64, nvalid, s);
    const int total = nseg * 4 * d.N * 32;
    k64_ion_maps<<<(total + 255) / 256, 256, 0, s>>>(P, L, d, Z, p.him);
    count_launch();
    for (int b0 = 0; b0 < B; b0 += bc) {
        const int nb = std::min(bc, B - b0);
        DW_CHECK(run_chunk64(p, d, nb, P, L, r + (int64_t)b0 * d.n * 3, R, Z, seg ? seg + b0 : nullptr,
                             nvalid, b0, lp + b0, phase ? phase + b0 : nullptr, E ? E + b0 : nullptr,
                             grad ? grad + (int64_t)b0 * 3 * d.n : nullptr, s));
    }
    return DW_OK;
}

}  // namespace dw

extern "C" {

// Test hook: FP64 determinant tangents (launch_tangents64) of nmat matrices with the 3 n + 1 derivative channels of
// MO [mat][3 n + 2][n][n]; K determinants per walker, nvalid (device, may be null) counts walkers. A scratch below
// dw_debug_det_tangents_fp64_bytes takes fewer matrices at a time, or the FP64 loop.
size_t dw_debug_det_tangents_fp64_bytes(int n, int nmat) { return dw::dets64_scratch_bytes(n, 3 * n + 2, nmat); }
int dw_debug_det_tangents_fp64(const double* MO, const double* Ainv, const double* sign, int n, int K, int nmat,
                               const int* nvalid, double* g, double* lapdet, void* scratch, size_t scratch_bytes, void* stream) {
    using namespace dw;
    reset_launch_count();
    if (!MO || !Ainv || !sign || !g || !lapdet || n < 1 || n > kMaxEl || K < 1 || nmat < 1 || nmat % K) return DW_ERR_ARG;
    Run64 q;
    q.d = Dims();
    q.d.n = n; q.d.K = K;
    q.C = 3 * n + 2; q.B = nmat / K; q.nvalid = nvalid;
    DW_CHECK(launch_tangents64(MO, Ainv, sign, q, nmat, g, lapdet, scratch, scratch_bytes, (cudaStream_t)stream));
    DW_CHECK_CUDA(cudaGetLastError());
    return DW_OK;
}

}  // extern "C"
