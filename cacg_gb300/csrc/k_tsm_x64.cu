// k_tsm_x64.cu -- FP64 tall x small products with fused updates on the fp16
// tensor cores (tcgen05, sm_103a), from exact digit planes (x64_util.cuh).
//
// Reference operations replaced (sclc/cacg), in FP64:
//   dense_distributedMatL_localMatR_Mul_v1  src/BLAS3.c:794-825  Q beta, Q alpha, AQ alpha
//   dense_mat_mat_add_TP                    src/BLAS3.c:579-612  Q = S - Q beta,
//                                                                 X += Q alpha, R -= AQ alpha
//
// Why: n k^2 FP64 FMAs keep the FP64 pipe (1.2 TFLOP/s) busy for most of an
// iteration.  Here a row of the tall operand shares one scale and a column of
// the small matrix another; the 34 digit-plane products with p + q <= 7 (one
// diagonal more than the Gram kernel: K terms average the dropped ones less
// than n rows do; K <= 144: every sum stays below 2^24, exact) run on the tensor
// cores, and the FP64 pipe is left with one conversion and one addition per output.
//
// The tall operand's columns may have any magnitudes (right-hand sides, columns
// of a block to factor), and FMAs do not mind: a scale per column commutes with
// them.  So does it here: column j goes by the power of two of about its norm
// (exponents e0, e1 of x64_col_exp), which the small matrix's row j gets instead.
// Both only shift digits, so the result for columns scaled by powers of two is the
// scaled result, bit for bit.  With norms b_j = 2^e_j the error of output column c is
// some 2^-54 of max_j b_j max_j b_j |W_jc|, b_j again 1 after the scaling, that is of
// the largest ||A_j|| |W_jc|: what FMAs leave, column by column.
//
// One persistent CTA of 17 or 21 warps per SM walks 128-row tiles of one column tile
// of NB <= 64 outputs:
//   * 8 (or 16) converter warps, 16 (8) rows each: read 32-column chunks of their rows, split
//     them into K-major plane tiles (double-buffered), and in passing read the
//     next tile's rows for their scales (that brings the tile into L2);
//   * one warp issues the MMAs against the small matrix's planes, which stay
//     in shared memory side by side in N (for Q and for AQ, where the X/R update's
//     two sets fit; else it is two launches), so plane p of the rows meets planes
//     0 .. 7-p in one or two wide MMAs; the accumulators of p + q = 0 .. 7 lie
//     side by side in tensor memory (two sets when they fit);
//   * 8 (or 4) epilogue warps, a row and half (all) its columns a thread, combine
//     the eight integer sums, scale them to FP64 and apply the update.
// Measured (before: the FMA kernels): Q update n = 884736, k = 96 13.5 -> 1.01 ms
// (the epilogue's FP64 conversions and the converters' integer work, each about
// half of the time's issue slots); X/R update m = 16 4.5 -> 0.65 ms; n = 65536,
// k = 128 1.89 -> 0.145 ms, m = 32 0.93 -> 0.139 ms; product error 1.3e-16 of the
// result (FMA chain 0.8e-16 to 1.1e-16), QR factors' error unchanged.  The column
// exponents cost 3 % of these (an addition an element, the small matrix's second set).
// A row with an Inf or NaN, or every row when the small matrix has one (or numbers
// whose scale leaves FP64's range), is formed by FP64 FMAs in the epilogue.  A wait
// that runs out sets kStatusTimeout.
#include <algorithm>
#include <cstdint>

#include "cacg_internal.cuh"
#include "tc5_util.cuh"
#include "x64_util.cuh"

namespace cacg {

constexpr int kXtM = 128;  // rows per tile
constexpr int kXtKC = 32;  // columns of the tall operand per step
// converter warps CW, epilogue warps EW (EW / 4 per tensor-memory lane
// quadrant), one issuing warp
constexpr int xt_epi_warps(int cw) { return cw == 16 ? 4 : 8; }
constexpr int xt_threads(int cw) { return 32 * (cw + xt_epi_warps(cw) + 1); }
constexpr unsigned kXtPlane = kXtM * kXtKC * 2;
constexpr unsigned kXtABytes = kXPlanes * kXtPlane;
constexpr int kXtMaxK = 144;
constexpr int kXtDiag = 8;  // accumulators: p + q = 0 .. 7

// kXtXR: X and R in one launch; kXtOne: one of them (part0)
enum { kXtQ = 0, kXtXR = 1, kXtMul = 2, kXtOne = 3 };
constexpr bool xt_is_xr(int mode) { return mode == kXtXR || mode == kXtOne; }

struct XtArgs {
    int64_t n;
    int K, N;               // tall operand columns, outputs
    const double *A0, *A1;  // tall operands (A1: the second product of the X/R update)
    const int *e0, *e1;     // their columns' exponents
    int part0;              // kXtOne: 0 X, 1 R
    int64_t lda;
    const double *W;  // K x N, row stride ldw
    int ldw;
    const double *C;  // kXtQ: S
    int64_t ldc;
    double *out;  // kXtQ: Q_new (may be C); kXtMul: the product
    int64_t ldo;
    double *X, *R, *S0;  // kXtXR (S0 may be NULL)
    int64_t lds;
    long long polls;  // limit of the pipeline's waits
    double *part;  // kXtXR: gridDim.x x N sums of squares of the new R (may be NULL)
    int *status;
};

// x's exponent field less its column's offset, in units of 2^-20
__device__ __forceinline__ int xt_key(double x, int f20) {
    return (int)((uint32_t)__double2hiint(x) & 0x7ff00000u) - f20;
}
// place of column j's offset: the eight that a converter lane needs for a 32-column
// chunk are contiguous (columns 8 u + 2 (lane % 4) + 0, 1)
__device__ __forceinline__ int xt_off(int j) {
    return (j & ~31) + 8 * ((j >> 1) & 3) + 2 * ((j >> 3) & 3) + (j & 1);
}
constexpr int kXtNoKey = INT32_MIN;
constexpr int kXtMaxExp = 1100;  // a row of finite values stays at 1023 or below
constexpr int kXtMinExp = 523;   // smaller rows (2^-500 of the columns' norms) share this scale
// row scales in shared memory: kXtFma no scale, | kXtFar results that may leave the normal numbers
constexpr int kXtFma = -1, kXtFar = 1 << 16;

template <bool VEC>
__device__ __forceinline__ double2 xt_load2(const double *p, int col, int K, bool rv) {
    double2 v = make_double2(0.0, 0.0);
    if constexpr (VEC) {
        if (rv && col < K) v = __ldg(reinterpret_cast<const double2 *>(p));
    } else {
        if (rv && col < K) v.x = __ldg(p);
        if (rv && col + 1 < K) v.y = __ldg(p + 1);
    }
    return v;
}

// VEC: K, lda even and A 16-byte aligned; OVEC: the same for the update's rows
template <int NC, int MODE, bool VEC, bool OVEC, int kXtConvWarps>
__global__ void __launch_bounds__(xt_threads(kXtConvWarps), 1) tsm_x64_kernel(XtArgs g) {
    constexpr int kXtEpiWarps = xt_epi_warps(kXtConvWarps), kEH = kXtEpiWarps / 4;
    constexpr int kXtThreads = xt_threads(kXtConvWarps);
    constexpr int kXtRG = kXtM / 8 / kXtConvWarps;  // 8-row groups per converter warp
    constexpr int NB = 16 * NC;
    constexpr int kAcc = kXtDiag * NB;            // accumulator columns of one tile
    constexpr int kBufs = 2 * kAcc <= 512 ? 2 : 1;  // accumulator sets
    constexpr int kTmem = kBufs * kAcc <= 256 ? 256 : 512;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // [A planes x2][W planes][row scales x2][column scales][operand column offsets][limits]
    // [mbarriers][tmem slot][abort]; W planes, scales, offsets and limits per operand
    constexpr int sets = MODE == kXtXR ? 2 : 1;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform, and known to be
    const int Kp = (g.K + 15) / 16 * 16;
    const int nchunk = (Kp + kXtKC - 1) / kXtKC;
    const unsigned sbo_b = (unsigned)(Kp / 8) * 128;
    unsigned char *wpl = smem_raw + 2 * kXtABytes;
    const unsigned w_bytes = (unsigned)(kXPlanes * NB / 8) * sbo_b;
    int *rowE = reinterpret_cast<int *>(wpl + (size_t)sets * w_bytes);
    int *colE = rowE + 2 * kXtM;    // NB a set
    int *offs = colE + sets * NB;   // 32 nchunk a set: the column's exponent less 1023, << 20
    int *lim = offs + sets * 32 * nchunk;  // 4 a set: smallest row scale, smallest and largest of colE
    uint64_t *sfull = reinterpret_cast<uint64_t *>(lim + 4 * sets);
    uint64_t *sfree = sfull + 2;
    uint64_t *tdone = sfree + 2;
    uint64_t *tfree = tdone + 2;
    uint64_t *rfull = tfree + 2;
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(rfull + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // sums of squares of this CTA's R values, by row of the tile and column
    constexpr int kSqP = NB + 1;
    double *sq = reinterpret_cast<double *>(tmem_slot + 2);

    const int c0 = blockIdx.y * NB;
    const int nc = min(NB, g.N - c0);
    const int64_t ntile = (g.n + kXtM - 1) / kXtM;
    const int mytiles =
        blockIdx.x < ntile ? (int)((ntile - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
    const int njobs = mytiles * sets;
    auto row0_of = [&](int job) {
        return (int64_t)((int)blockIdx.x + job / sets * (int)gridDim.x) * kXtM;
    };
    auto set_of = [&](int job) { return job % sets; };

    // ---- the small matrix's planes, one scale per column
    for (int i = tid; i < sets * NB; i += kXtThreads) colE[i] = kXtNoKey;
    for (int i = tid; i < sets * 32 * nchunk; i += kXtThreads) {
        const int t = i / (32 * nchunk), j = i - t * 32 * nchunk;
        offs[t * 32 * nchunk + xt_off(j)] = j < g.K ? ((t ? g.e1 : g.e0)[j] - 1023) * (1 << 20) : 0;
    }
    if (xt_is_xr(MODE) && g.part)
        for (int i = tid; i < kXtM * kSqP; i += kXtThreads) sq[i] = 0.0;
    if (tid == 0) {
        for (int x = 0; x < 2; ++x) {
            t5_mbar_init(&sfull[x], kXtConvWarps);
            t5_mbar_init(&sfree[x], 1);
            t5_mbar_init(&tdone[x], 1);
            t5_mbar_init(&tfree[x], kXtEpiWarps);
            t5_mbar_init(&rfull[x], kXtConvWarps);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         t5_smem_u32(tmem_slot)),
                     "r"(kTmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    // its values go through the A planes' space (K x NB, zeros past its ends)
    double *ws = reinterpret_cast<double *>(smem_raw);
#pragma unroll 4
    for (int e = tid; e < Kp * NB; e += kXtThreads) {
        const int j = e / NB, c = e % NB;
        ws[e] = j < g.K && c < nc ? g.W[(size_t)j * g.ldw + c0 + c] : 0.0;
    }
    __syncthreads();
    bool wbad = false;
    auto wexp = [](double x) { return (int)(((uint32_t)__double2hiint(x) >> 20) & 0x7ffu); };
    auto off = [&](int t, int j) { return offs[t * 32 * nchunk + xt_off(j)] >> 20; };
    if (tid < kXtThreads / NB * NB) {
        const int c = tid % NB;
        int mx[2] = {kXtNoKey, kXtNoKey};
        for (int j = tid / NB; j < Kp; j += kXtThreads / NB) {
            const double x = ws[j * NB + c];
            if (x64_key(x) == 0u) continue;
            const int ex = wexp(x);
            wbad |= ex == 0x7ff;
            mx[0] = max(mx[0], max(ex, 1) + off(0, j));
            if (sets == 2) mx[1] = max(mx[1], max(ex, 1) + off(1, j));
        }
        atomicMax(&colE[c], mx[0]);
        if (sets == 2) atomicMax(&colE[NB + c], mx[1]);
    }
    __syncthreads();
    if (warp < sets) {
        // a zero's shift is at least 64 at every row scale: it has no significand bits
        int lo = INT32_MAX, cmin = INT32_MAX, cmax = INT32_MIN;
        for (int i = lane; i < 32 * nchunk; i += 32) lo = min(lo, offs[warp * 32 * nchunk + i] >> 20);
        for (int i = lane; i < NB; i += 32) {
            int &e = colE[warp * NB + i];
            if (e == kXtNoKey) e = 1023;
            cmin = min(cmin, e);
            cmax = max(cmax, e);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        cmin = __reduce_min_sync(0xffffffffu, cmin);
        cmax = __reduce_max_sync(0xffffffffu, cmax);
        if (lane == 0) {
            lim[4 * warp] = lo;
            lim[4 * warp + 1] = cmin;
            lim[4 * warp + 2] = cmax;
        }
    }
    __syncthreads();
    for (int e = tid; e < sets * (Kp / 2) * NB; e += kXtThreads) {
        const int t = e >= Kp / 2 * NB, ee = e - t * (Kp / 2 * NB);
        const int j = 2 * (ee / NB), c = ee % NB;
        double x[2];
        uint32_t E20[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            x[u] = ws[(j + u) * NB + c];
            int E = colE[t * NB + c] - off(t, j + u);
            if (wexp(x[u]) == 0) {  // 0, or so small that its column's scale has to drop it
                wbad |= x[u] != 0.0 && E < 64;
                x[u] = 0.0;
                E = 64;
            }
            E20[u] = (uint32_t)E << 20;
        }
        uint32_t w[kXPlanes];
        x64_planes2(x[0], x[1], E20[0], E20[1], w);
#pragma unroll
        for (int p = 0; p < kXPlanes; ++p) {
            const int nn = p * NB + c;
            *reinterpret_cast<uint32_t *>(wpl + t * w_bytes + (nn >> 3) * sbo_b + (j >> 3) * 128 +
                                          (nn & 7) * 16 + (j & 7) * 2) = w[p];
        }
    }
    t5_fence_proxy_async();
    t5_fence_before();
    const bool wide = __syncthreads_or(wbad) != 0;  // every row by FMAs
    t5_fence_after();
    const unsigned tmem = *tmem_slot;

    if (warp < kXtConvWarps) {
        // ------------------------------------------------------ converters
        // lane: row lane / 4 of each of the warp's 8-row groups, column pair
        // lane % 4 of each octet
        const int lr = lane >> 2, lc = 2 * (lane & 3);
        const int noct = Kp / 8;
        auto row_ptr = [&](int job, int rg, bool &rv) {
            const int64_t row = row0_of(job) + 8 * (kXtRG * warp + rg) + lr;
            rv = row < g.n;
            const double *A = set_of(job) ? g.A1 : g.A0;
            return A + (rv ? row : 0) * g.lda + lc;
        };
        // offsets of this lane's columns, eight a chunk
        auto off_of = [&](int job) { return offs + set_of(job) * 32 * nchunk + 4 * lc; };
        auto pair_max = [&](int k) {
            k = max(k, __shfl_xor_sync(0xffffffffu, k, 1));
            return max(k, __shfl_xor_sync(0xffffffffu, k, 2));
        };
        int key[kXtRG];
        bool rv[kXtRG], rvn[kXtRG];
        const double *pa[kXtRG], *pn[kXtRG];
        double2 cur[kXtRG][4];
#pragma unroll
        for (int rg = 0; rg < kXtRG; ++rg) {
            key[rg] = kXtNoKey;
            rvn[rg] = false;
            pa[rg] = pn[rg] = row_ptr(0, rg, rv[rg]);
            for (int o = 0; o < noct; ++o) {
                const double2 v = xt_load2<VEC>(pa[rg] + 8 * o, 8 * o + lc, g.K, rv[rg]);
                const int2 f = *reinterpret_cast<const int2 *>(offs + xt_off(8 * o + lc));
                key[rg] = max(key[rg], max(xt_key(v.x, f.x), xt_key(v.y, f.y)));
            }
            key[rg] = pair_max(key[rg]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                cur[rg][u] = xt_load2<VEC>(pa[rg] + 8 * u, 8 * u + lc, g.K, rv[rg]);
        }
        bool ok = true;
        int step = 0;
        for (int job = 0; job < njobs && ok; ++job) {
            const int x = (int)(job & 1);
            if (job >= 2) {
                ok = __all_sync(0xffffffffu, t5_mbar_wait_or_abort(
                                                 &tfree[x], (unsigned)(((job >> 1) - 1) & 1),
                                                 abort_flag, g.polls));
                if (!ok) break;
            }
            const bool more = job + 1 < njobs;
            const int set = set_of(job);
            const int *offc = off_of(job), *offn = off_of(job + 1);
            int E[kXtRG];
            // the rows of two jobs on, into L2: the scan of the next job's rows below
            // has only a few hundred instructions to hide its loads behind
            if (job + 2 < njobs) {
#pragma unroll
                for (int rg = 0; rg < kXtRG; ++rg) {
                    bool rp;
                    const double *q = row_ptr(job + 2, rg, rp) - lc;
                    if (rp)
                        for (int b = 64 * lc; b < g.K * 8; b += 512)
                            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(
                                reinterpret_cast<const char *>(q) + b));
                }
            }
#pragma unroll
            for (int rg = 0; rg < kXtRG; ++rg) {
                E[rg] = max(key[rg] >> 20, max(64 - lim[4 * set], kXtMinExp));
                // not far: sums between 1 and 2^79 times 2^(E + colE - 2114) are normal numbers
                const bool far = E[rg] + lim[4 * set + 1] < 1114 || E[rg] + lim[4 * set + 2] > 3014;
                if (lc == 0)
                    rowE[x * kXtM + 8 * (kXtRG * warp + rg) + lr] =
                        wide || E[rg] > kXtMaxExp ? kXtFma : far ? E[rg] | kXtFar : E[rg];
                if (more) pn[rg] = row_ptr(job + 1, rg, rvn[rg]);
                key[rg] = kXtNoKey;
            }
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(&rfull[x]);
            for (int ch = 0; ch < nchunk; ++ch, ++step) {
                const int b = (int)(step & 1);
                const bool lastc = ch + 1 == nchunk;
                if (step >= 2) {
                    ok = __all_sync(0xffffffffu, t5_mbar_wait_or_abort(
                                                     &sfree[b], (unsigned)(((step >> 1) - 1) & 1),
                                                     abort_flag, g.polls));
                    if (!ok) break;
                }
                int fc[8];
                auto offs8 = [&](const int *p, int(&f)[8]) {
                    const int4 a = *reinterpret_cast<const int4 *>(p + 32 * ch);
                    const int4 b = *reinterpret_cast<const int4 *>(p + 32 * ch + 4);
                    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
                    f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
                };
                offs8(offc, fc);
#pragma unroll
                for (int rg = 0; rg < kXtRG; ++rg) {
                    // the next job's rows: their scales
                    double2 nxt[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int o = 4 * ch + u;
                        nxt[u] = xt_load2<VEC>(pn[rg] + 8 * o, 8 * o + lc, g.K,
                                               more && rvn[rg] && o < noct);
                    }
                    unsigned char *dst = smem_raw + b * kXtABytes + (kXtRG * warp + rg) * 512 +
                                         lr * 16 + lc * 2;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int o = 4 * ch + u;
                        if (o < noct) {
                            const double2 v = cur[rg][u];
                            if (!lastc)
                                cur[rg][u] = xt_load2<VEC>(pa[rg] + 8 * (o + 4), 8 * (o + 4) + lc,
                                                           g.K, rv[rg] && o + 4 < noct);
                            const uint32_t E20 = (uint32_t)E[rg] << 20;
                            uint32_t w[kXPlanes];
                            x64_planes2(v.x, v.y, E20 + fc[2 * u], E20 + fc[2 * u + 1], w);
#pragma unroll
                            for (int p = 0; p < kXPlanes; ++p)
                                *reinterpret_cast<uint32_t *>(dst + p * kXtPlane + u * 128) = w[p];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        int2 f = make_int2(fc[2 * u], fc[2 * u + 1]);
                        if constexpr (sets == 2)
                            f = *reinterpret_cast<const int2 *>(offn + 32 * ch + 2 * u);
                        key[rg] = max(key[rg], max(xt_key(nxt[u].x, f.x), xt_key(nxt[u].y, f.y)));
                    }
                }
                t5_fence_proxy_async();
                __syncwarp();
                if (lane == 0) t5_mbar_arrive(&sfull[b]);
            }
            if (!ok) break;
#pragma unroll
            for (int rg = 0; rg < kXtRG; ++rg) {
                key[rg] = pair_max(key[rg]);
                pa[rg] = pn[rg];
                rv[rg] = rvn[rg];
                if (more) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        cur[rg][u] = xt_load2<VEC>(pa[rg] + 8 * u, 8 * u + lc, g.K, rv[rg]);
                }
            }
        }
        if (!ok && lane == 0) *abort_flag = 1;
    } else if (warp < kXtConvWarps + kXtEpiWarps) {
        // -------------------------------------------------------- epilogue
        // column groups of 4: half, half + kEH, ...
        const int quad = warp & 3, half = (warp >> 2) & (kEH - 1);
        const int rt = 32 * quad + lane;
        bool ok = true;
        for (int job = 0; job < njobs && ok; ++job) {
            const int x = (int)(job & 1);
            const unsigned ph = (unsigned)((job >> 1) & 1);
            const int set = set_of(job), part = MODE == kXtOne ? g.part0 : set;
            const int *ce = colE + set * NB;
            const int64_t row = row0_of(job) + rt;
            const bool rv = row < g.n;
            // the addend's row: the update reads it, then writes the result in place
            const double *src = nullptr;
            if constexpr (MODE == kXtQ) src = g.C + row * g.ldc + c0;
            if constexpr (xt_is_xr(MODE)) src = (part ? g.R : g.X) + row * g.N + c0;
            if (src && rv && half == 0)
                for (int b = 0; b < nc * 8; b += 128)
                    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(
                        reinterpret_cast<const char *>(src) + b));
            ok = __all_sync(0xffffffffu,
                            t5_mbar_wait_or_abort(&rfull[x], ph, abort_flag, g.polls) &&
                                t5_mbar_wait_or_abort(&tdone[x], ph, abort_flag, g.polls));
            if (!ok) break;
            t5_fence_after();
            const int re = rowE[x * kXtM + rt], E = re & (kXtFar - 1);
            const unsigned ta = tmem + ((unsigned)(32 * quad) << 16) +
                                (unsigned)((kBufs == 2 ? x : 0) * kAcc);
            auto addend = [&](int c, double (&s)[4]) {
                if constexpr (MODE != kXtMul) {
                    if constexpr (OVEC) {
#pragma unroll
                        for (int q = 0; q < 4; q += 2) {
                            double2 v = make_double2(0.0, 0.0);
                            if (rv && c + q < nc) v = *reinterpret_cast<const double2 *>(src + c + q);
                            s[q] = v.x;
                            s[q + 1] = v.y;
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) s[q] = rv && c + q < nc ? src[c + q] : 0.0;
                    }
                }
            };
            double ad[2][4];
            addend(4 * half, ad[0]);
            addend(4 * half + 4 * kEH, ad[1]);
#pragma unroll
            for (int ci = 0; ci < NB / (4 * kEH); ++ci) {
                const int cc = 4 * (kEH * ci + half);
                unsigned r[kXtDiag][4];
                __syncwarp();
#pragma unroll
                for (int d = 0; d < kXtDiag; ++d) t5_ld4_nowait(ta + d * NB + cc, r[d]);
                t5_wait_ld();
                double s[4], v[4];
                int sc[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = ad[ci & 1][q];
                if (ci + 2 < NB / (4 * kEH)) addend(cc + 8 * kEH, ad[ci & 1]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    int D[kXtDiag];
#pragma unroll
                    for (int d = 0; d < kXtDiag; ++d) D[d] = __float2int_rn(__uint_as_float(r[d][q]));
                    // |D[d]| <= (d + 1) K 2^14: the int products fit; h 2^32 + l in units of 2^40
                    const long long h =
                        (long long)(D[0] * 256 + D[1]) * 65536 + (long long)(D[2] * 256 + D[3]);
                    const long long l = (long long)(D[4] * 16777216ll) +
                                        ((long long)D[5] * 65536 + (long long)D[6] * 256 + D[7]);
                    sc[q] = E + ce[cc + q] - (2154 - 40);
                    v[q] = x64_join(h, l);
                }
                if (re < kXtFar) {
                    // h 2^32 and l may cancel: the sum is what is zero (and 1 or more if not)
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        v[q] = x64_scaled(v[q], __double2hiint(v[q]) == 0, sc[q]);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {  // by halves: overflow and underflow as FP64's
                        const int s2 = min(max(sc[q], -2000), 2000), h = s2 >> 1;
                        v[q] = v[q] * __hiloint2double((1023 + h) << 20, 0) *
                               __hiloint2double((1023 + s2 - h) << 20, 0);
                    }
                }
                if (re == kXtFma && rv) {  // no scale for this row: FP64 FMAs
                    const double *a = (set ? g.A1 : g.A0) + row * g.lda;
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = 0.0;
                    for (int j = 0; j < g.K; ++j) {
                        const double aj = a[j];
                        const double *w = g.W + (size_t)j * g.ldw + c0 + cc;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (cc + q < nc) v[q] = fma(aj, w[q], v[q]);
                    }
                }
                double o[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    o[q] = MODE == kXtMul ? v[q]
                           : (xt_is_xr(MODE) && part == 0) ? s[q] + v[q]
                                                           : s[q] - v[q];
                auto put = [&](double *dst) {
                    if constexpr (OVEC) {
#pragma unroll
                        for (int q = 0; q < 4; q += 2)
                            if (cc + q < nc)
                                *reinterpret_cast<double2 *>(dst + cc + q) =
                                    make_double2(o[q], o[q + 1]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (cc + q < nc) dst[cc + q] = o[q];
                    }
                };
                if (!rv) {
                } else if constexpr (xt_is_xr(MODE)) {
                    put((part ? g.R : g.X) + row * g.N + c0);
                    if (part && g.S0) put(g.S0 + row * g.lds + c0);
                    if (part && g.part) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            double &t = sq[rt * kSqP + cc + q];
                            t = fma(o[q], o[q], t);
                        }
                    }
                } else {
                    put(g.out + row * g.ldo + c0);
                }
            }
            t5_fence_before();
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(&tfree[x]);
        }
        if (!ok && lane == 0) *abort_flag = 1;
    } else {
        // ------------- MMA issuer: a whole warp, one elected lane at the MMAs
        int step = 0, last = -1;
        bool ok = true;
        for (int job = 0; job < njobs && ok; ++job) {
            const int x = (int)(job & 1);
            // the accumulator set's previous tile has been read
            if (kBufs == 2 && job >= 2)
                ok = t5_mbar_wait_or_abort(&tfree[x], (unsigned)(((job >> 1) - 1) & 1), abort_flag,
                                           g.polls);
            if (kBufs == 1 && job >= 1)
                ok = t5_mbar_wait_or_abort(&tfree[x ^ 1], (unsigned)(((job - 1) >> 1) & 1),
                                           abort_flag, g.polls);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            for (int ch = 0; ch < nchunk; ++ch, ++step) {
                const int b = (int)(step & 1);
                ok = __all_sync(0xffffffffu, t5_mbar_wait_or_abort(
                                                 &sfull[b], (unsigned)((step >> 1) & 1), abort_flag,
                                                 g.polls));
                if (!ok) break;
                t5_fence_after();
                const unsigned abase = t5_smem_u32(smem_raw + b * kXtABytes);
                const unsigned bbase = t5_smem_u32(wpl) + set_of(job) * w_bytes;
                const unsigned dset = tmem + (kBufs == 2 ? x : 0) * kAcc;
                const int nk = min(2, Kp / 16 - 2 * ch);
                if (t5_elect()) {
                    for (int kk = 0; kk < nk; ++kk) {
                        const unsigned first = (ch == 0 && kk == 0) ? 0u : 1u;
                        const unsigned bk = bbase + (4 * ch + 2 * kk) * 128;
                        // accumulators [d0, d0 + nd) of plane p with planes d0 - p ..: at
                        // most 256 columns an MMA
                        auto run = [&](int p, int d0, int nd, unsigned acc) {
                            const uint64_t ad = t5_desc(abase + p * kXtPlane + kk * 256, 512);
                            const unsigned bp = bk + (unsigned)((d0 - p) * (NB / 8)) * sbo_b;
                            const int N = nd * NB;
                            t5_mma(dset + d0 * NB, ad, t5_desc(bp, sbo_b),
                                   x64_idesc(kXtM, N < 256 ? N : 256), acc);
                            if (N > 256)
                                t5_mma(dset + d0 * NB + 256, ad, t5_desc(bp + 32 * sbo_b, sbo_b),
                                       x64_idesc(kXtM, N - 256), acc);
                        };
                        run(0, 0, 7, first);
                        run(1, 1, 6, 1u);
                        run(1, 7, 1, first);
#pragma unroll
                        for (int p = 2; p < kXPlanes; ++p) run(p, p, kXtDiag - p, 1u);
                    }
                    t5_commit(&sfree[b]);
                    if (ch + 1 == nchunk) t5_commit(&tdone[x]);
                }
                __syncwarp();
                last = step;
            }
        }
        if (!ok && lane == 0) *abort_flag = 1;
        // every committed MMA finishes before tensor memory goes, and every commit's
        // arrival lands before the barriers do (bounded)
        if (last >= 0) t5_mbar_wait(&sfree[last & 1], (unsigned)((last >> 1) & 1));
        const int done = (last + 1) / nchunk - 1;  // the last job whose last chunk was issued
        if (done >= 0) t5_mbar_wait(&tdone[done & 1], (unsigned)((done >> 1) & 1));
    }
    t5_fence_before();
    const int gave_up = __syncthreads_or(*abort_flag);
    if (warp == 0) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                     "r"(kTmem));
    }
    if (gave_up && tid == 0 && g.status) atomicOr(g.status, kStatusTimeout);
    if (xt_is_xr(MODE) && g.part) {
        // columns in row order: 8 threads a column sum 16 rows each, then in order
        const int c = tid >> 3, h = tid & 7;
        double t = 0.0;
        if (c < NB)
            for (int r = 0; r < kXtM / 8; ++r) t += sq[(h * (kXtM / 8) + r) * kSqP + c];
        double all = 0.0;
        for (int i = 0; i < 8; ++i) all += __shfl_sync(0xffffffffu, t, (lane & ~7) + i);
        if (h == 0 && c < nc) g.part[(size_t)blockIdx.x * g.N + c0 + c] = all;
    }
}

// ------------------------------------------------------------------- host
static size_t xt_smem(int K, int NB, int sets) {
    const int Kp = (K + 15) / 16 * 16;
    return 2 * (size_t)kXtABytes + 2 * kXtM * sizeof(int) + 10 * 8 + 16 +
           sets * ((size_t)(kXPlanes * NB / 8) * (Kp / 8) * 128 +
                   (size_t)(NB + (Kp + 31) / 32 * 32 + 4) * 4);
}
static size_t xt_sq_bytes(int NB) { return (size_t)kXtM * (NB + 1) * sizeof(double); }

// *blocks (kXtXR): the CTAs that wrote g.part, 0 when shared memory had no room
// for the sums and the caller forms the norms from R
template <int MODE>
static int xt_launch(cudaStream_t st, XtArgs g, int *blocks = nullptr) {
    if (g.n <= 0) return CACG_OK;
    if (g.K <= 0 || g.K > kXtMaxK || g.N <= 0 || !g.e0) return CACG_ERR_UNSUPPORTED;
    g.polls = pipeline_wait_limit();
    const int maxsm = (int)max_smem_optin();
    int tn = (g.N + 63) / 64, NB;
    for (;; ++tn) {
        NB = ((g.N + tn - 1) / tn + 15) / 16 * 16;
        if (xt_smem(g.K, NB, 1) <= (size_t)maxsm || NB == 16) break;
    }
    size_t smem = xt_smem(g.K, NB, MODE == kXtXR ? 2 : 1);
    if constexpr (MODE == kXtXR) {
        if (NB > 32 || smem + xt_sq_bytes(NB) > (size_t)maxsm) {
            // the small matrix's planes for Q and for AQ do not fit side by side: two
            // launches (K = 128, N = 32, n = 65536: 138 us; narrower column tiles would
            // convert Q and AQ twice)
            XtArgs x = g, r = g;
            x.part = nullptr;
            r.part0 = 1;
            r.A0 = g.A1;
            r.e0 = g.e1;
            const int rc = xt_launch<kXtOne>(st, x);
            return rc != CACG_OK ? rc : xt_launch<kXtOne>(st, r, blocks);
        }
    }
    if (smem > (size_t)maxsm) return CACG_ERR_UNSUPPORTED;
    if (g.part && smem + xt_sq_bytes(NB) <= (size_t)maxsm)
        smem += xt_sq_bytes(NB);
    else
        g.part = nullptr;
    tn = (g.N + NB - 1) / NB;
    const int64_t tiles = (g.n + kXtM - 1) / kXtM;
    const int64_t gx = std::max<int64_t>(1, std::min<int64_t>(tiles, std::max(1, sm_count() / tn)));
    const dim3 grid((unsigned)gx, (unsigned)tn);
    if (blocks) *blocks = g.part ? (int)gx : 0;
    const bool vec = g.K % 2 == 0 && g.lda % 2 == 0 && aligned16(g.A0) &&
                     (MODE != kXtXR || aligned16(g.A1));
    bool ovec = g.N % 2 == 0;
    if (xt_is_xr(MODE))
        ovec = ovec && aligned16(g.X) && aligned16(g.R) &&
               (!g.S0 || (aligned16(g.S0) && g.lds % 2 == 0));
    else
        ovec = ovec && aligned16(g.out) && g.ldo % 2 == 0 &&
               (MODE == kXtMul || (aligned16(g.C) && g.ldc % 2 == 0));
    // the converters' work grows with K, the epilogue's with NB.  X/R update,
    // n = 884736, K = 96, NB = 16: 768 us with 16 + 4 warps, 900 with 8 + 8;
    // n = 262144, K = 64, NB = 16: 164 and 179; n = 65536, K = 128, NB = 32: 138 and
    // 158.  Q update, n = 884736, K = 96, NB = 48: 1340 against 1262.
    constexpr int kMany = xt_is_xr(MODE) ? 16 : 8;
    const bool many = xt_is_xr(MODE) && g.K >= 4 * NB;
#define XT_GO(NC, V, O, CW)                                                          \
    do {                                                                             \
        set_smem_attr(tsm_x64_kernel<NC, MODE, V, O, CW>, maxsm);                    \
        tsm_x64_kernel<NC, MODE, V, O, CW><<<grid, xt_threads(CW), smem, st>>>(g);   \
    } while (0)
#define XT_CASE(NC)                             \
    case NC:                                    \
        if constexpr ((MODE == kXtXR && NC > 2) || (MODE == kXtOne && NC < 2)) { \
            return CACG_ERR_UNSUPPORTED;        \
        } else if (vec && many) {               \
            if (ovec)                           \
                XT_GO(NC, true, true, kMany);   \
            else                                \
                XT_GO(NC, true, false, kMany);  \
        } else if (vec) {                       \
            if (ovec)                           \
                XT_GO(NC, true, true, 8);       \
            else                                \
                XT_GO(NC, true, false, 8);      \
        } else {                                \
            XT_GO(NC, false, false, 8);         \
        }                                       \
        break;
    switch (NB / 16) {
        XT_CASE(1)
        XT_CASE(2)
        XT_CASE(3)
        XT_CASE(4)
        default:
            return CACG_ERR_UNSUPPORTED;
    }
#undef XT_CASE
#undef XT_GO
    return check_launch();
}

int launch_qupdate_x64(cudaStream_t st, int64_t n, int k, double *Qout, int64_t ldo,
                       const double *Qin, int64_t ldq, const int *qexp, const double *S,
                       int64_t lds, const double *beta, int *status) {
    if ((const void *)Qout == (const void *)Qin) return CACG_ERR_ARG;
    XtArgs g{};
    g.n = n, g.K = k, g.N = k;
    g.A0 = Qin, g.lda = ldq, g.e0 = qexp;
    g.W = beta, g.ldw = k;
    g.C = S, g.ldc = lds;
    g.out = Qout, g.ldo = ldo;
    g.status = status;
    return xt_launch<kXtQ>(st, g);
}

int launch_xrupdate_x64(cudaStream_t st, int64_t n, int k, int m, const double *Q,
                        const double *AQ, int64_t ldq, const int *qexp, const int *aqexp,
                        const double *alpha, double *X, double *R, double *S0, int64_t lds,
                        double *norms, double *ws, int *status) {
    XtArgs g{};
    g.n = n, g.K = k, g.N = m;
    g.A0 = Q, g.A1 = AQ, g.lda = ldq, g.e0 = qexp, g.e1 = aqexp;
    g.W = alpha, g.ldw = m;
    g.X = X, g.R = R, g.S0 = S0, g.lds = lds;
    g.status = status;
    g.part = norms ? ws : nullptr;
    int blocks = 0;
    const int rc = xt_launch<kXtXR>(st, g, &blocks);
    if (rc != CACG_OK || !norms) return rc;
    if (blocks > 0) return launch_colsum(st, ws, blocks, m, norms);
    return launch_colnorm(st, n, m, R, norms, ws);
}

int launch_tallsmall_x64(cudaStream_t st, int64_t n, int K, int N, const double *A, int64_t lda,
                         const int *aexp, const double *W, int ldw, double *Y, int64_t ldy, int *status) {
    XtArgs g{};
    g.n = n, g.K = K, g.N = N;
    g.A0 = A, g.lda = lda, g.e0 = aexp;
    g.W = W, g.ldw = ldw;
    g.out = Y, g.ldo = ldy;
    g.status = status;
    return xt_launch<kXtMul>(st, g);
}

}  // namespace cacg
