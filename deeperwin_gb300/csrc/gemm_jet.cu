// Persistent tcgen05 GEMM of the tangent passes: the T = 3 n_el + 2 channel rows of each electron
// (value, gradients, Laplacian) times the weights, with the forward-Laplacian tanh fused (layers) or
// the envelope orbitals (backflow: the Slater channels are written directly, not the backflow).
//
//   Y[(e, t), f] = epilogue( sum_k A[(e, t), k] W[f, k] )
//
// * A and W are BF16 (NP = 1) or split-BF16 (NP = 2: x = hi + lo, three MMAs per K step, FP32
//   accumulation in TMEM).
// * The product is formed transposed: the 128 TMEM lanes are features, the columns are channel rows.
//   An epilogue thread then owns one feature of all T channels of an electron, so the tanh, the sum of
//   squared gradient rows and the coefficients of the jet stay in its registers (no exchange between
//   lanes or warps, one tanh per electron and feature), and an electron needs no padding to a power of
//   two: its rows start at a multiple of 8 columns (a swizzle atom) in a tile of up to 256.
// * With more than 128 features two CTAs form a pair (cta_group::2): 256 features x up to 256 rows, each
//   CTA with the weights of 128 features resident in shared memory (160 KB at K = 320 in two parts) and
//   half of the rows in its ring. That halves the ring bytes per MMA, and the MMAs (N = 224 of 256 at 16
//   electrons) read less shared memory per product: single CTAs with N = 112 and the same ring were
//   held at two thirds of this rate by the MMAs' operand reads and the two-stage ring's round trips,
//   whether or not the pair shared its loads by multicast. Up to 128 features run on single CTAs with
//   256 rows (h_map, Jastrow).
// * Units (feature blocks, tile) are split evenly and in order over the SMs, whole electrons per tile.
// * Warp roles (576 threads): warp 0 = TMA producer, warp 1 = MMA issuer, warps 2-17 = epilogue, two
//   sets of four (one warp per TMEM lane quarter) for each of the two accumulator buffers. The sixteen
//   warps are what the epilogue needs: its instructions are few, but a warp's own chain is long (with
//   eight warps the same kernel took 1.6 times as long). Stores go straight from registers: a warp
//   writes 32 consecutive features of a row (64 bytes per BF16 part, whole sectors).
// Bound by HBM: the layer of 16 electrons (K = 320, 409,600 rows) moves 943 MB in 204 us (4.6 TB/s, 69 %
// of the measured copy rate; before, with rows as TMEM lanes, electrons padded to 64 rows and the jet
// exchanged through shared memory, 390 us for the same rows), h_map (K = 256) 515 MB in 86 us (6.0 TB/s).
// The envelope in the backflow's epilogue replaces a kernel that read the backflow back: backflow and
// envelopes of a C2H4 local energy (4,096 walkers) 6.4 -> 4.0 ms, of 512 walkers at 40 electrons 23.1 ->
// 13.4 ms; at 10 electrons and 10 ions, where a thread's envelope costs as much as its channels, 2.2 -> 2.35.
// Every mbarrier wait is bounded; on timeout the kernel records an error flag, stops issuing, waits
// (bounded) for its TMA loads in flight, frees its TMEM and returns.
#include "gemm_tc.cuh"
#include <algorithm>
#include <type_traits>

// lambdas that hold accumulator registers by reference: called out of line they would go through local memory
#define DW_INLINE __attribute__((always_inline))

namespace dw {

namespace {

constexpr int BM = 128;                              // features per block (TMEM lanes)
constexpr int kTileRows = 256;                       // channel rows (TMEM columns) of a tile
constexpr int BK = 64;                               // K-columns per stage (128-byte swizzled rows)
constexpr int kBufs = 512 / kTileRows;               // accumulator buffers
constexpr int kSets = 4;                             // epilogue warp sets, kSets / kBufs per buffer
constexpr int kThreads = 64 + 128 * kSets;
constexpr int kBufCols = kTileRows;                  // TMEM columns of a buffer
constexpr int kLdRb = 256;                           // row pitch of the row bias (the layer width)
constexpr int kMaxStages = 8;
constexpr int kSmemMax = 226 * 1024;                 // dynamic shared memory of a CTA at most (1 KB aligned)

struct JetArgs {
    int NF, K, nk;                                   // features, reduction width, stages per tile
    int fpb;                                         // features per block (at most 128)
    int T, Tq, ept, ncol;                            // channel rows, their column pitch, electrons per tile, MMA N
    int n, ns, i0;                                   // electrons per walker; those taken: [i0, i0 + ns)
    int E;                                           // electrons in all (walkers * ns)
    int ntiles;
    int64_t units;                                   // feature blocks * tiles
    int stages;                                      // ring depth
    uint32_t x_part, w_part;                         // bytes of one part of a stage, of a weight slab
    int single_load;                                 // a tile's rows are consecutive and unpadded
    int64_t rows;
    const float* bias; const float* rowbias;
    void* C;
    EnvEpi env;
    int* error;
};
enum Epilogue { kTanh, kEnvelope };

// Position in the list of units.
struct Unit {
    int group, tile;
    __device__ Unit(int64_t u, int ntiles) : group((int)(u / ntiles)), tile((int)(u % ntiles)) {}
    __device__ void next(int ntiles) { if (++tile == ntiles) { tile = 0; ++group; } }
};

// An electron's T accumulator columns, 16 at a time: mid(v, c) for every chunk but the last, last(v, c)
// for that one. The next chunk's load is in flight while a chunk is worked on.
template <class Mid, class Last>
__device__ __forceinline__ void for_chunks(uint32_t col0, int T, Mid mid, Last last) {
    float A[16], B[16];
    const int lastc = (T - 1) / 16;
    tmem_ld16(col0, A);
    for (int c = 0;;) {
        tmem_wait_ld16(A);
        if (c == lastc) { last(A, c); break; }
        tmem_ld16(col0 + 16 * (c + 1), B);
        mid(A, c);
        ++c;
        tmem_wait_ld16(B);
        if (c == lastc) { last(B, c); break; }
        tmem_ld16(col0 + 16 * (c + 1), A);
        mid(B, c);
        ++c;
    }
    __syncwarp();
}

// Store of feature f of a row at o (row pitch LDC columns; split rows are [hi | lo]).
template <int OUT, int LDC> struct RowOut;
template <int LDC> struct RowOut<0, LDC> {
    using T = float;
    static constexpr int pitch = LDC;
    __device__ static __forceinline__ void put(T* o, float x) { *o = x; }
};
template <int LDC> struct RowOut<1, LDC> {
    using T = __nv_bfloat16;
    static constexpr int pitch = LDC;
    __device__ static __forceinline__ void put(T* o, float x) { *o = __float2bfloat16_rn(x); }
};
template <int LDC> struct RowOut<2, LDC> {
    using T = __nv_bfloat16;
    static constexpr int pitch = 2 * LDC;
    __device__ static __forceinline__ void put(T* o, float x) {
        const __nv_bfloat16 hi = __float2bfloat16_rn(x);
        o[0] = hi;
        o[LDC] = __float2bfloat16_rn(x - __bfloat162float(hi));
    }
};

// The forward-Laplacian tanh of one feature over an electron's channels, a chunk at a time:
//   y0 = tanh(z0), y_t = d1 z_t, y_lap = d1 z_lap - 2 y0 d1 sum_t z_t^2, d1 = 1 - y0^2.
// The squares are added over 8 channels in order, then pairwise up to 32 channels, then in order.
template <int OUT, int LDC>
struct Jet {
    using Row = RowOut<OUT, LDC>;
    float y0 = 0.f, d1 = 0.f, sum = 0.f, half = 0.f;
    // channels t0 .. t0 + NV - 1; the electron has rem = T - t0 channels from t0 on (LAST: rem <= NV)
    template <int NV, bool FIRST, bool LAST>
    __device__ __forceinline__ void chunk(float (&v)[16], int c, int rem, float bias, bool fok, typename Row::T* o) {
        if (FIRST) {
            v[0] += bias;
            y0 = tanhf(v[0]);
            d1 = 1.f - y0 * y0;
        }
        float b8[2] = {0.f, 0.f};
        #pragma unroll
        for (int j = 0; j < NV; ++j) {
            float sq = __fmul_rn(v[j], v[j]);
            if ((FIRST && j == 0) || (LAST && j >= rem - 1)) sq = 0.f;
            b8[j / 8] = __fadd_rn(b8[j / 8], sq);
        }
        const float pair = __fadd_rn(b8[0], b8[1]);
        if ((c & 1) == 0) half = pair;
        if ((c & 1) || LAST) {
            const float s32 = (c & 1) ? __fadd_rn(half, pair) : half;
            sum = c < 2 ? s32 : __fadd_rn(sum, s32);
        }
        if (!fok) return;
        const float cl = -2.f * y0 * d1 * sum;
        #pragma unroll
        for (int j = 0; j < NV; ++j) {
            // (a branch on j == rem - 1 would index v dynamically, through local memory)
            float y = LAST ? fmaf(d1, v[j], j == rem - 1 ? cl : 0.f) : d1 * v[j];
            if (FIRST && j == 0) y = fmaf(0.f, v[j], y0);
            if (!LAST || j < rem) Row::put(o + j * Row::pitch, y);
        }
    }
};

// Electron i of walker b against the ions, ion `lane` per lane: difference vector and distance
// (negative: no such ion, or padding of a packed geometry) and its reciprocal.
struct Geo {
    float s0, s1, s2, dd, inv;
};
// x / b from the correctly rounded reciprocal of b (P. W. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: the quotient is correctly rounded
// too, barring underflow): one reciprocal per (electron, ion) serves all orbital columns.
__device__ __forceinline__ float quotient(float x, float b, float inv) {
    const float q = x * inv;
    return fmaf(fmaf(-q, b, x), inv, q);
}
__device__ __forceinline__ Geo geometry(const EnvEpi& p, int b, int i, int lane) {
    const Dims& d = p.d;
    Geo g{0.f, 0.f, 0.f, -1.f, -1.f};
    if (lane < d.N) {
        const float* ri = p.r + ((int64_t)b * d.n + i) * 3;
        const int I = seg_of(d, b) * d.N + lane;
        g.s0 = ri[0] - p.R[I * 3]; g.s1 = ri[1] - p.R[I * 3 + 1]; g.s2 = ri[2] - p.R[I * 3 + 2];
        g.dd = p.Z[I] > 0 ? sqrtf(g.s0 * g.s0 + g.s1 * g.s1 + g.s2 * g.s2) : -1.f;
        g.inv = 1.f / g.dd;
    }
    return g;
}
// The envelope of one orbital column (envelope_orbitals.py:96-127): value, gradient and Laplacian in
// r_i. Called by a whole warp; two ions at a time, added in order.
struct EnvValue {
    float e, g[3], lap;
};
__device__ __forceinline__ EnvValue envelope_of(const EnvEpi& p, const Geo& geo, int col) {
    const Dims& d = p.d;
    float env = 0.f, g[3] = {0.f, 0.f, 0.f}, lapv = 0.f;
    for (int I0 = 0; I0 < d.N; I0 += 2) {
        float s0[2], s1[2], s2[2], dd[2], e[2], gs[2], q[2];
        #pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int I = min(I0 + u, d.N - 1);
            s0[u] = __shfl_sync(0xffffffffu, geo.s0, I);
            s1[u] = __shfl_sync(0xffffffffu, geo.s1, I);
            s2[u] = __shfl_sync(0xffffffffu, geo.s2, I);
            dd[u] = __shfl_sync(0xffffffffu, geo.dd, I);
            const float inv = __shfl_sync(0xffffffffu, geo.inv, I);
            const float a = __ldg(p.sp_alpha + I * d.KN + col);
            e[u] = __ldg(p.wts + I * d.KN + col) * expf(-a * dd[u]);
            gs[u] = quotient(-a * e[u], dd[u], inv);
            q[u] = __fsub_rn(__fmul_rn(a, a), quotient(2.f * a, dd[u], inv));
        }
        #pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (I0 + u >= d.N || dd[u] < 0.f) continue;
            env += e[u];
            g[0] = fmaf(gs[u], s0[u], g[0]); g[1] = fmaf(gs[u], s1[u], g[1]); g[2] = fmaf(gs[u], s2[u], g[2]);
            lapv = fmaf(e[u], q[u], lapv);
        }
    }
    return EnvValue{env, {g[0], g[1], g[2]}, lapv};
}

// OUT: 0 = fp32, 1 = bf16, 2 = split-BF16. EPI: forward-Laplacian tanh (C with row pitch LDC), or the
// envelope (Slater channels). CG: CTAs per MMA. With CG = 2 a cluster of two
// CTAs forms 256 features x 256 rows: each keeps the weights of 128 features and loads half of the
// rows, so a stage is half as large for the same work; CTA 0 issues the MMAs, and the barriers it
// waits on (full, wfull, tempty) count both CTAs.
template <int NP, int OUT, int EPI, int LDC, int CG>
__global__ void __launch_bounds__(kThreads, 1)
k_gemm_jet(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
           const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1, JetArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int S = a.stages, nk = a.nk;
    const uint32_t w_part = a.w_part, x_part = a.x_part;   // one part of a K slab of the weights / of a stage
    uint8_t* ring = smem + (size_t)nk * NP * w_part;
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + (size_t)S * NP * x_part);
    uint64_t* empty = full + kMaxStages;
    uint64_t* tfull = empty + kMaxStages;            // [kBufs]
    uint64_t* tempty = tfull + kBufs;
    uint64_t* wfull = tempty + kBufs;
    uint64_t* wempty = wfull + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wempty + 1);
    __shared__ int s_err, s_set_err[kSets];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        s_err = 0;
        for (int h = 0; h < kSets; ++h) s_set_err[h] = 0;
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int h = 0; h < kBufs; ++h) { mbar_init(&tfull[h], 1); mbar_init(&tempty[h], CG * 4 * kSets / kBufs); }
        mbar_init(wfull, 1);
        mbar_init(wempty, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 0) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();                     // the peer's barriers are initialised, its TMEM allocated
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0;
    const uint32_t lead = lane == 0;                 // the lane that issues copies and MMAs
    // this CTA's (pair's) units: (group of CG feature blocks, tile)
    const int64_t nc = gridDim.x / CG, ci = blockIdx.x / CG;
    const int64_t u0 = a.units * ci / nc, u1 = a.units * (ci + 1) / nc;
    const int ept = a.ept;                           // electrons per tile and CTA

    if (warp == 0) {
        // ring position: stage s, and the parity of the consumer's last release of it
        int s = 0;
        uint32_t par = 1, fills = 0, nw = 0;
        bool err = false;
        int wblk = -1;
        const uint32_t tx = (uint32_t)(CG * NP * ept * a.T * BK * 2);
        const int nload = a.single_load ? 1 : ept;
        Unit w(u0, a.ntiles);
        for (int64_t u = u0; u < u1 && !err; ++u, w.next(a.ntiles)) {
            const int blk = w.group * CG + rank, k0 = (w.tile * CG + rank) * ept;
            const int b0 = k0 / a.ns, j0 = k0 % a.ns;
            if (blk != wblk) {                       // weights of the next feature block, once the last one is used up
                if (nw > 0 && !mbar_wait_warp(wempty, (nw - 1) & 1)) { err = true; break; }
                if (rank == 0) mbar_expect_tx(wfull, (uint32_t)(CG * nk * NP) * w_part, lead);
                for (int kt = 0; kt < nk; ++kt) {
                    uint8_t* dst = smem + (size_t)(kt * NP) * w_part;
                    if (CG == 2) {
                        tma_load_2d_pair(dst, &tmW0, cta0_addr(wfull), kt * BK, blk * a.fpb, lead);
                        if (NP == 2) tma_load_2d_pair(dst + w_part, &tmW1, cta0_addr(wfull), kt * BK, blk * a.fpb, lead);
                    } else {
                        tma_load_2d(dst, &tmW0, wfull, kt * BK, blk * a.fpb, lead);
                        if (NP == 2) tma_load_2d(dst + w_part, &tmW1, wfull, kt * BK, blk * a.fpb, lead);
                    }
                }
                wblk = blk;
                ++nw;
            }
            for (int kt = 0; kt < nk; ++kt) {
                if (!mbar_wait_warp(&empty[s], par)) { err = true; break; }
                if (rank == 0) mbar_expect_tx(&full[s], tx, lead);
                const uint32_t full0 = CG == 2 ? cta0_addr(&full[s]) : 0;
                uint8_t* st = ring + (size_t)s * NP * x_part;
                int row = (b0 * a.n + a.i0 + j0) * a.T, j = j0, k = k0;
                for (int e = 0; e < nload; ++e) {
                    if (k >= a.E) row = (int)a.rows;             // past the end: zeros
                    uint8_t* dst = st + e * a.Tq * (BK * 2);
                    if (CG == 2) {
                        tma_load_2d_pair(dst, &tmA0, full0, kt * BK, row, lead);
                        if (NP == 2) tma_load_2d_pair(dst + x_part, &tmA1, full0, kt * BK, row, lead);
                    } else {
                        tma_load_2d(dst, &tmA0, &full[s], kt * BK, row, lead);
                        if (NP == 2) tma_load_2d(dst + x_part, &tmA1, &full[s], kt * BK, row, lead);
                    }
                    row += a.T;
                    ++k;
                    if (++j == a.ns) { j = 0; row += (a.n - a.ns) * a.T; }
                }
                fills = min(fills + 1, (uint32_t)S);
                if (++s == S) { s = 0; par ^= 1; }
            }
        }
        if (err) {
            if (lead) atomicExch(&s_err, 1);
            if (rank == 0) {
                if (nw > 0) mbar_wait_warp(wfull, (nw - 1) & 1);
                // the last fill of each stage: before s in this turn of the ring, from s on in the last
                for (uint32_t k = 0; k < fills; ++k) mbar_wait_warp(&full[k], (int)k < s ? par ^ 1 : par);
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = idesc_bf16(CG * a.ncol, CG * BM);
            int s = 0;
            uint32_t par = 0, it = 0, nw = 0;
            bool err = false;
            int wblk = -1;
            Unit w(u0, a.ntiles);
            for (int64_t u = u0; u < u1 && !err; ++u, ++it, w.next(a.ntiles)) {
                const uint32_t acc = it % kBufs;
                if (w.group != wblk) {
                    if (nw > 0) {                    // every MMA on the last block's weights is done
                        if (CG == 2) umma_commit_pair(wempty, lead);
                        else umma_commit(wempty, lead);
                    }
                    if (!mbar_wait_warp(wfull, nw & 1)) { err = true; break; }
                    wblk = w.group;
                    ++nw;
                }
                if (!mbar_wait_warp(&tempty[acc], ((it / kBufs) & 1) ^ 1)) { err = true; break; }
                tc_fence_after();
                const uint32_t d = tmem + acc * kBufCols;
                for (int kt = 0; kt < nk; ++kt) {
                    if (!mbar_wait_warp(&full[s], par)) { err = true; break; }
                    tc_fence_after();
                    const uint8_t* wp = smem + (size_t)(kt * NP) * w_part;
                    const uint8_t* xp = ring + (size_t)s * NP * x_part;
                    const uint64_t w0 = smem_desc<BK>(wp), x0 = smem_desc<BK>(xp);
                    const uint64_t w1 = smem_desc<BK>(wp + (NP - 1) * w_part), x1 = smem_desc<BK>(xp + (NP - 1) * x_part);
                    #pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        const uint64_t o = (uint64_t)(kk * 2);
                        auto mma = [&](uint64_t x, uint64_t y, uint32_t accum) {
                            if (CG == 2) umma_bf16_pair(d, x + o, y + o, idesc, accum, lead);
                            else umma_bf16(d, x + o, y + o, idesc, accum, lead);
                        };
                        mma(w0, x0, (kt | kk) ? 1u : 0u);
                        if (NP == 2) {
                            mma(w1, x0, 1u);
                            mma(w0, x1, 1u);
                        }
                    }
                    if (CG == 2) umma_commit_pair(&empty[s], lead);
                    else umma_commit(&empty[s], lead);
                    if (++s == S) { s = 0; par ^= 1; }
                }
                if (CG == 2) umma_commit_pair(&tfull[acc], lead);
                else umma_commit(&tfull[acc], lead);
            }
            if (err && lead) atomicExch(&s_err, 1);
        }
    } else {
        // TMEM lane quarter, warp set: the two sets of a buffer take alternate electrons
        const int q = warp & 3, h = (warp - 2) >> 2, buf = h % kBufs;
        const int T = a.T;
        using Row = RowOut<OUT, LDC>;
        uint32_t it = 0;
        Unit w(u0, a.ntiles);
        for (int64_t u = u0; u < u1; ++u, ++it, w.next(a.ntiles)) {
            if ((int)(it % kBufs) != buf) continue;
            const int blk = w.group * CG + rank, k0 = w.tile * CG * ept;
            const int f = blk * a.fpb + q * 32 + lane;
            const bool fok = q * 32 + lane < a.fpb && f < a.NF;
            // geometry of the set's first electron, fetched while the accumulator is finished
            Geo geo{0.f, 0.f, 0.f, -1.f, -1.f};
            auto fetch = [&](int e) {
                const int k = k0 + e, b = k / a.ns;
                if (e < CG * ept && k < a.E) geo = geometry(a.env, b, a.i0 + k - b * a.ns, lane);
            };
            if (EPI == kEnvelope) fetch(h / kBufs);
            const bool ready = mbar_wait(&tfull[buf], (it / kBufs) & 1);
            if (!ready && lane == 0) s_set_err[h] = 1;
            asm volatile("bar.sync %0, 128;" ::"r"(1 + h) : "memory");      // the set agrees before leaving
            if (*(volatile int*)&s_set_err[h]) { if (lane == 0) atomicExch(&s_err, 1); break; }
            tc_fence_after();
            if (q * 32 < a.fpb && blk * a.fpb + q * 32 < a.NF) {
                const float bias = EPI == kTanh && a.bias && fok ? __ldg(a.bias + f) : 0.f;
                for (int e = h / kBufs; e < CG * ept && k0 + e < a.E; e += kSets / kBufs) {
                    const int k = k0 + e, b = k / a.ns, i = a.i0 + k - b * a.ns;
                    const uint32_t col0 = tmem + ((uint32_t)(q * 32) << 16) + buf * kBufCols +
                                          (CG == 2 && e >= ept ? a.ncol + (e - ept) * a.Tq : e * a.Tq);
                    if constexpr (EPI == kEnvelope) {
                        const Dims& d = a.env.d;
                        const EnvValue ev = envelope_of(a.env, geo, min(f, a.NF - 1));
                        fetch(e + kSets / kBufs);                    // the next electron's, behind this one's stores
                        const int n2 = d.n * d.n, ko = f / d.n, own = 1 + 3 * i;
                        float* mo = a.env.MO + ((int64_t)b * d.K + ko) * T * n2 + i * d.n + f - ko * d.n;
                        float bf0 = 0.f, bo[3] = {0.f, 0.f, 0.f};    // backflow value and own-coordinate rows
                        // rem: channels from 16 c on (the last chunk has the Laplacian at rem - 1)
                        auto general = [&](const float (&v)[16], int c, int rem) DW_INLINE {
                            #pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                if (j >= rem) break;
                                float x = ev.e * v[j];
                                const unsigned o3 = (unsigned)(16 * c + j - own);
                                if (o3 < 3u) {
                                    x = fmaf(o3 == 0 ? ev.g[0] : (o3 == 1 ? ev.g[1] : ev.g[2]), bf0, x);
                                    if (o3 == 0) bo[0] = v[j];
                                    else if (o3 == 1) bo[1] = v[j];
                                    else bo[2] = v[j];
                                } else if (j == rem - 1 && 16 * c + j == T - 1) {
                                    x = fmaf(ev.lap, bf0, x);
                                    #pragma unroll
                                    for (int k3 = 0; k3 < 3; ++k3) x = fmaf(2.f * ev.g[k3], bo[k3], x);
                                }
                                mo[j * n2] = x;
                            }
                        };
                        for_chunks(col0, T,
                            [&](const float (&v)[16], int c) DW_INLINE {
                                if (c == 0) bf0 = v[0];
                                if (!fok) return;
                                if (own >= 16 * (c + 1) || own + 3 <= 16 * c) {
                                    #pragma unroll
                                    for (int j = 0; j < 16; ++j) mo[j * n2] = ev.e * v[j];
                                } else {
                                    general(v, c, 16);
                                }
                                mo += 16 * n2;
                            },
                            [&](const float (&v)[16], int c) DW_INLINE {
                                if (c == 0) bf0 = v[0];
                                if (fok) general(v, c, T - 16 * c);
                            });
                    } else {
                        // the row bias of the next chunk is fetched while this one is worked on
                        const bool has_rb = a.rowbias && fok;
                        const float* rb = has_rb ? a.rowbias + (int64_t)b * T * kLdRb + f : nullptr;
                        typename Row::T* o = static_cast<typename Row::T*>(a.C) + (int64_t)(b * a.n + i) * T * Row::pitch + f;
                        float rv[16];
                        auto load_rb = [&](int t0) DW_INLINE {
                            if (t0 + 16 <= T) {
                                #pragma unroll
                                for (int j = 0; j < 16; ++j) rv[j] = has_rb ? __ldg(rb + j * kLdRb) : 0.f;
                            } else {
                                #pragma unroll
                                for (int j = 0; j < 16; ++j) rv[j] = has_rb && t0 + j < T ? __ldg(rb + j * kLdRb) : 0.f;
                            }
                            rb += 16 * kLdRb;
                        };
                        load_rb(0);
                        Jet<OUT, LDC> jet;
                        using std::integral_constant;
                        using std::true_type;
                        using std::false_type;
                        auto step = [&](float (&v)[16], auto nv, auto first, auto last, int c) DW_INLINE {
                            constexpr int NV = decltype(nv)::value;
                            #pragma unroll
                            for (int j = 0; j < NV; ++j) v[j] += rv[j];
                            if (!decltype(last)::value) load_rb(16 * (c + 1));
                            jet.template chunk<NV, decltype(first)::value, decltype(last)::value>(v, c, T - 16 * c, bias, fok, o);
                            o += 16 * Row::pitch;
                        };
                        const integral_constant<int, 16> n16;
                        const integral_constant<int, 8> n8;
                        for_chunks(col0, T,
                            [&](float (&v)[16], int c) DW_INLINE {
                                if (c == 0) step(v, n16, true_type(), false_type(), c);
                                else step(v, n16, false_type(), false_type(), c);
                            },
                            [&](float (&v)[16], int c) DW_INLINE {
                                if (c == 0) step(v, n16, true_type(), true_type(), c);
                                else if (T - 16 * c > 8) step(v, n16, false_type(), true_type(), c);
                                else step(v, n8, false_type(), true_type(), c);
                            });
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) mbar_arrive_cluster(cta0_addr(&tempty[buf]));
                else mbar_arrive(&tempty[buf]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();                     // no MMA, copy or arrival of the pair is left
    if (s_err && threadIdx.x == 0) atomicExch(a.error, 1);
    if (warp == 0) {
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

template <int NP, int OUT, int EPI, int LDC, int CG>
int launch_jet_cg(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C,
                  const JetRows& r, int NF, int K, const GemmEpi& epi, const EnvEpi* env, cudaStream_t s) {
    if (r.nw <= 0 || r.ns <= 0) return DW_OK;
    if (r.T < 1 || r.T > 128 || NF <= 0 || K <= 0 || (epi.rowbias && epi.ldrb != kLdRb)) return DW_ERR_ARG;
    JetArgs a;
    a.NF = NF; a.K = K; a.nk = (K + BK - 1) / BK;
    a.T = r.T; a.Tq = round_up(r.T, 8);
    a.n = r.n; a.ns = r.ns; a.i0 = r.i0; a.E = r.nw * r.ns;
    a.rows = (int64_t)r.nw * r.n * r.T;
    a.single_load = a.T == a.Tq && a.ns == a.n;
    a.bias = epi.bias; a.rowbias = epi.rowbias;
    a.C = C;
    if (env) a.env = *env;
    a.error = tc_error_flag();
    if (!a.error) return DW_ERR_CUDA;
    // A part of a stage: whole 1024-byte swizzle atoms of 8 rows; the MMA reads ncol rows. A part of a
    // weight slab holds only the features there are: the MMA's other rows read what follows it (the
    // ring, 128 rows of 128 bytes or more), into accumulator lanes that nothing uses.
    const int w_rows = std::min(BM, round_up(NF, 8));
    a.w_part = w_rows * BK * 2;
    const int w_bytes = a.nk * NP * a.w_part, fixed = 1024 + 512;
    // 256 rows per tile; 128 on a single CTA whose weights leave less than two stages of 256 (65 to 128
    // features at K = 256)
    int stage = 0;
    for (int cap = kTileRows / CG; cap >= 128; cap -= 128) {
        // the last electron's chunks of 16 columns end within the buffer
        const int last = round_up(a.T, 16);
        for (a.ept = cap / a.Tq;; --a.ept) {
            a.ncol = round_up(a.ept * a.Tq, 16);
            if ((CG - 1) * a.ncol + (a.ept - 1) * a.Tq + last <= kBufCols) break;
        }
        a.x_part = a.ncol * BK * 2;
        stage = NP * a.x_part;
        a.stages = std::min(kMaxStages, (kSmemMax - fixed - w_bytes) / stage);
        if (a.stages >= 2) break;
    }
    if (a.stages < 2) return DW_ERR_ARCH;
    a.ntiles = (a.E + CG * a.ept - 1) / (CG * a.ept);
    // the features spread evenly over the blocks, so that the CTAs of a pair have equal epilogues
    const int groups = (NF + CG * BM - 1) / (CG * BM);
    a.fpb = round_up((NF + groups * CG - 1) / (groups * CG), 8);
    a.units = (int64_t)a.ntiles * groups;
    const int Kp = round_up(K, 64), box = a.single_load ? a.ept * a.T : a.T;
    CUtensorMap ma0, ma1, mw0, mw1;
    DW_CHECK(make_map(&ma0, A, a.rows, K, (int64_t)NP * lda, BK, box, false));
    DW_CHECK(make_map(&mw0, W0, NF, K, Kp, BK, w_rows, false));
    ma1 = ma0; mw1 = mw0;
    if (NP == 2) {
        DW_CHECK(make_map(&ma1, A + lda, a.rows, K, (int64_t)NP * lda, BK, box, false));
        DW_CHECK(make_map(&mw1, W1, NF, K, Kp, BK, w_rows, false));
    }
    const size_t smem = (size_t)fixed + w_bytes + (size_t)a.stages * stage;
    auto kern = k_gemm_jet<NP, OUT, EPI, LDC, CG>;
    DW_CHECK_CUDA(allow_smem(kern, kSmemMax));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * std::min<int64_t>(a.units, num_sms() / CG)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = CG; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = CG > 1 ? 1 : 0;
    DW_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ma0, ma1, mw0, mw1, a));
    count_launch();
    return DW_OK;
}

template <int NP, int OUT, int EPI, int LDC>
int launch_jet(const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C, const JetRows& r, int NF,
               int K, const GemmEpi& epi, const EnvEpi* env, cudaStream_t s) {
    const __nv_bfloat16* a = reinterpret_cast<const __nv_bfloat16*>(A);
    // pairs of CTAs where there is more than one block of 128 features
    if (NF > BM) return launch_jet_cg<NP, OUT, EPI, LDC, 2>(a, lda, W0, W1, C, r, NF, K, epi, env, s);
    return launch_jet_cg<NP, OUT, EPI, LDC, 1>(a, lda, W0, W1, C, r, NF, K, epi, env, s);
}

}  // namespace

int gemm_jet(int np, int out, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, void* C,
             int ldc, const JetRows& r, int NF, int K, const GemmEpi& epi, cudaStream_t s) {
    // row pitches of the layer input (320), the Jastrow layers (64) and h_map (32)
    if (np == 2 && out == 2 && ldc == 320) return launch_jet<2, 2, kTanh, 320>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    if (np == 2 && out == 2 && ldc == 64) return launch_jet<2, 2, kTanh, 64>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    if (np == 2 && out == 0 && ldc == 32) return launch_jet<2, 0, kTanh, 32>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    if (np == 1 && out == 1 && ldc == 320) return launch_jet<1, 1, kTanh, 320>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    if (np == 1 && out == 1 && ldc == 64) return launch_jet<1, 1, kTanh, 64>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    if (np == 1 && out == 0 && ldc == 32) return launch_jet<1, 0, kTanh, 32>(A, lda, W0, W1, C, r, NF, K, epi, nullptr, s);
    return DW_ERR_ARG;
}

int gemm_jet_env(int np, const void* A, int lda, const __nv_bfloat16* W0, const __nv_bfloat16* W1, const JetRows& r, int K,
                 const EnvEpi& env, cudaStream_t s) {
    const int NF = env.d.KN;
    if (np == 2) return launch_jet<2, 0, kEnvelope, 1>(A, lda, W0, W1, nullptr, r, NF, K, GemmEpi(), &env, s);
    if (np == 1) return launch_jet<1, 0, kEnvelope, 1>(A, lda, W0, W1, nullptr, r, NF, K, GemmEpi(), &env, s);
    return DW_ERR_ARG;
}

}  // namespace dw

extern "C" {

// Test hook: gemm_jet on split-BF16 rows (np = 2); out 0 (fp32) or 2 (split-BF16).
int dw_debug_gemm_jet(int out, const void* A, int lda, const void* W0, const void* W1, void* C, int ldc, int nw,
                      int n, int T, int ns, int i0, int NF, int K, const float* bias, const float* rowbias, void* stream) {
    using namespace dw;
    if (!tc_available()) return DW_ERR_UNSUPPORTED;
    GemmEpi e;
    e.bias = bias; e.rowbias = rowbias; e.ldrb = 256; e.Tp = T;
    return gemm_jet(2, out, A, lda, (const __nv_bfloat16*)W0, (const __nv_bfloat16*)W1, C, ldc,
                    JetRows{nw, n, T, ns, i0}, NF, K, e, (cudaStream_t)stream);
}

// The same on BF16 rows (np = 1); out 0 (fp32) or 1 (bf16).
int dw_debug_gemm_jet_bf16(int out, const void* A, int lda, const void* W, void* C, int ldc, int nw, int n, int T, int ns,
                           int i0, int NF, int K, const float* bias, const float* rowbias, void* stream) {
    using namespace dw;
    if (!tc_available()) return DW_ERR_UNSUPPORTED;
    GemmEpi e;
    e.bias = bias; e.rowbias = rowbias; e.ldrb = 256; e.Tp = T;
    return gemm_jet(1, out, A, lda, (const __nv_bfloat16*)W, nullptr, C, ldc, JetRows{nw, n, T, ns, i0}, NF, K, e,
                    (cudaStream_t)stream);
}

// Test hook: gemm_jet_env, the backflow of electrons [i0, i0 + ns) of nw walkers of n electrons and N ions (geometry
// seg[b] of nseg, seg may be null) times the envelope, into MO [walker][dets][3 n + 2][n][n].
int dw_debug_gemm_jet_env(int np, const void* A, int lda, const void* W0, const void* W1, const float* r, const float* R,
                          const int32_t* Z, const int32_t* seg, int nseg, const float* alpha, const float* weights, float* MO,
                          int nw, int n, int N, int dets, int ns, int i0, int K, void* stream) {
    using namespace dw;
    if (!tc_available()) return DW_ERR_UNSUPPORTED;
    if (n < 1 || n > kMaxEl || N < 1 || N > kMaxIons || dets < 1 || i0 < 0 || i0 + ns > n || nseg < 1) return DW_ERR_ARG;
    EnvEpi env{r, R, Z, alpha, weights, MO, Dims()};
    env.d.n = n; env.d.N = N; env.d.K = dets; env.d.KN = dets * n; env.d.T = env.d.Tp = 3 * n + 2;
    env.d.seg = seg; env.d.nseg = nseg;
    return gemm_jet_env(np, A, lda, (const __nv_bfloat16*)W0, (const __nv_bfloat16*)W1, JetRows{nw, n, env.d.T, ns, i0}, K, env,
                        (cudaStream_t)stream);
}

}  // extern "C"
