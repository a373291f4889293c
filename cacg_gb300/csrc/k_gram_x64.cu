// k_gram_x64.cu -- FP64 Gram products C = L^T [R1 | R2] on the fp16 tensor
// cores (tcgen05, sm_103a), from exact digit planes.
//
// Reference operations replaced (sclc/cacg): distributedMatLTransposeMatRMul
// (src/BLAS3.c:699-726) and distributedMatLTransposeMatRMul_updated
// (src/BLAS3.c:730-758) in FP64, with the allreduce that follows each.
//
// Why: this part's FP64 pipe gives 1.2 TFLOP/s, 1/1600 of its fp16 tensor
// rate, and an FP64 FMA Gram keeps it 96 % busy; 28 fp16 digit-plane products
// (x64_util.cuh) do the same sum 20 times faster.
//
// Accuracy.  A digit holds an element to 2^-56 of the power of two M above its
// column's largest in the row chunk, so a row's product is within 2^-53 M_a M_b
// (the roundings and the dropped planes; 2^-58 is usual), whatever the product's
// own size.  An FMA chain's error goes with sum |L||R|, and that can be far
// smaller: rows graded against each other, one large element a column.  So the
// planes are for chunks where it is not.  With D_a the sum over the rows of
// log2(M_a / |L_ra|), the arithmetic-geometric mean inequality gives
//     sum_r |L_ra||R_rb| >= rows M_a M_b 2^-(D_a + D_b)/rows
// and a chunk with (max D_a + max D_b) / rows above kXgSpread is summed by FP64
// FMAs.  (A zero has no error in its row; counting kXgSpread bits for it keeps the
// bound true for the rows left.)  The planes' error is then below 2^(kXgSpread - 53) of
// sum |L||R|, and about 2^(kXgSpread - 58) / sqrt(rows) of it in practice: 2^-49 at 64
// rows, 2^-52 at 6000, at the line.  Normal data stays at 8 to 10 bits.
//
// The solvers ask for less (normwise): their Gram matrices have to be accurate to
// ||L_a|| ||R_b||, since that is what the factorisation and the updates keep, and their
// blocks have columns of up to 17 bits (varying coefficients, 32 right-hand sides) and
// far more (point sources).  M_a <= 2 ||L_a||, so the planes give that without the line:
// about 2^-57 for spread columns, 2^-51 where one element of 6000 rows carries both.
// Point sources, alone and beside spread right-hand sides, tolerances to 1e-12: the
// iterations and residuals of the FMA Gram, in 13 to 29 % of the time.
//
// Two or three launches:
//   colmax   the largest magnitude and the sum of the logarithms of every column
//            over each row chunk (a column's digits share one scale per chunk);
//            small operands are scanned by the product kernel itself;
//   gram     split-K over row chunks, one CTA of 17 warps per SM: 16 converter
//            warps copy 32-row steps to shared memory (cp.async into slots
//            that only the copying thread reads: no barrier), split them into
//            digit planes (MN-major core matrices, double-buffered) and one
//            warp issues the MMAs.  The B planes are stacked side by side in
//            the MMA's N dimension and the accumulators of p + q = 0 .. 6 lie
//            side by side in tensor memory, so plane p of A is multiplied with
//            planes 0 .. 6-p of B by one or two wide MMAs: A is read from
//            shared memory 10 times a step instead of 28.  After 128 rows the
//            integer sums (below 2^24, exact) are folded into integer
//            registers (64 + 24 bits per output, exact), and scaled to FP64
//            once per chunk.  A chunk over the line above, or with Inf, NaN or a
//            column below 2^-959, is summed by the same CTA's FP64 FMAs instead;
//   reduce   sums the chunks' FP64 partials in a fixed order (and recomputes the
//            outputs should a wait of the product kernel have run out).
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "cacg_internal.cuh"
#include "tc5_util.cuh"
#include "x64_util.cuh"

namespace cacg {

constexpr int kXgKT = 32;                          // rows per step
constexpr int kXgM = 128;                          // MMA M (L columns, zero-padded)
constexpr int kXgGroup = 4;                        // steps per accumulation group (128 rows)
constexpr int kXgConvWarps = 16;
constexpr int kXgThreads = 32 * kXgConvWarps + 32;  // + the MMA issuer's warp
constexpr int kXgSpread = 12;  // bits: see above
constexpr int kXgNoLine = INT32_MAX;
constexpr int kXgMaxUnits = 6;  // (8 columns, 8 rows) units per warp and step
constexpr int kXgMaxStages = 4;  // steps of raw rows in flight
constexpr unsigned kXgABytes = kXPlanes * kXgM * kXgKT * 2;  // A planes of one step

struct XgOperands {
    const double *L, *R1, *R2;
    int64_t ldl, ldr1, ldr2;
    int ka, kb1, kb2;
};

// ------------------------------------------------------------ column maxima
// Sums of a column's logarithms, in units of 2^-8 (the key's exponent and first
// mantissa bits: at most log2 |x| + 1023), and its zeros beside them
constexpr int kXgZeroBit = 42;
__device__ __forceinline__ uint64_t xg_log(uint32_t key) {
    return key == 0u ? 1ull << kXgZeroBit : (uint64_t)(key >> 12);
}
// such sums added up in shared memory by 32-bit parts (a 64-bit shared addition is a
// loop: 64 threads of a column take it for 30 us a launch)
struct XgLogSum {
    uint32_t lo, hi, zeros;
};
__device__ __forceinline__ void xg_add(XgLogSum &t, uint64_t s) {
    const uint64_t l = s & ((1ull << kXgZeroBit) - 1);
    atomicAdd(&t.lo, (uint32_t)l & 0xfffffu);
    atomicAdd(&t.hi, (uint32_t)(l >> 20));
    if (s >> kXgZeroBit) atomicAdd(&t.zeros, (uint32_t)(s >> kXgZeroBit));
}
__device__ __forceinline__ uint64_t xg_logs(const XgLogSum &t) {
    return ((uint64_t)t.hi << 20) + t.lo;
}

// emax, elog[(chunk * sub + s) * (ka + kb) + column]: block (chunk, s) covers the
// s-th part of the chunk's rows (LOG: the logarithms too)
template <bool VEC, bool LOG>
__global__ void __launch_bounds__(512)
    gram_x64_colmax_kernel(int64_t n, int64_t rows_per_chunk, int64_t rows_per_sub, XgOperands o,
                           uint32_t *__restrict__ emax, unsigned long long *__restrict__ elog) {
    __shared__ uint32_t mx[3 * 256];
    __shared__ XgLogSum lg[LOG ? 3 * 256 : 1];
    const int kc = o.ka + o.kb1 + o.kb2;
    for (int i = threadIdx.x; i < kc; i += blockDim.x) {
        mx[i] = 0u;
        if constexpr (LOG) lg[i] = XgLogSum{0u, 0u, 0u};
    }
    __syncthreads();
    const int64_t c0 = (int64_t)blockIdx.x * rows_per_chunk;
    const int64_t rb = c0 + (int64_t)blockIdx.y * rows_per_sub;
    const int64_t re = min(min(n, c0 + rows_per_chunk), rb + rows_per_sub);
    int base = 0;
    for (int t = 0; t < 3; ++t) {
        const double *p = t == 0 ? o.L : t == 1 ? o.R1 : o.R2;
        const int64_t ld = t == 0 ? o.ldl : t == 1 ? o.ldr1 : o.ldr2;
        const int w = t == 0 ? o.ka : t == 1 ? o.kb1 : o.kb2;
        if (w > 0) {
            const int tpr = VEC ? w / 2 : w;
            const int rpb = blockDim.x / tpr;
            const int r = threadIdx.x / tpr, c = (threadIdx.x % tpr) * (VEC ? 2 : 1);
            if (r < rpb) {
                uint32_t k0 = 0u, k1 = 0u;
                uint64_t s0 = 0, s1 = 0;
#pragma unroll 8
                for (int64_t row = rb + r; row < re; row += rpb) {
                    if constexpr (VEC) {
                        const double2 v = __ldg(reinterpret_cast<const double2 *>(p + row * ld + c));
                        const uint32_t e0 = x64_key(v.x), e1 = x64_key(v.y);
                        k0 = max(k0, e0);
                        k1 = max(k1, e1);
                        if constexpr (LOG) s0 += xg_log(e0), s1 += xg_log(e1);
                    } else {
                        const uint32_t e0 = x64_key(__ldg(p + row * ld + c));
                        k0 = max(k0, e0);
                        if constexpr (LOG) s0 += xg_log(e0);
                    }
                }
                atomicMax(&mx[base + c], k0);
                if constexpr (VEC) atomicMax(&mx[base + c + 1], k1);
                if constexpr (LOG) {
                    xg_add(lg[base + c], s0);
                    if constexpr (VEC) xg_add(lg[base + c + 1], s1);
                }
            }
        }
        base += w;
    }
    __syncthreads();
    const size_t out = ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * kc;
    for (int i = threadIdx.x; i < kc; i += blockDim.x) {
        emax[out + i] = mx[i];
        if constexpr (LOG) elog[out + i] = xg_logs(lg[i]) | (uint64_t)lg[i].zeros << kXgZeroBit;
    }
}

// -------------------------------------------------------------- the products
__device__ __forceinline__ void xg_cp16(void *smem, const void *g, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(t5_smem_u32(smem)), "l"(g),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void xg_cp8(void *smem, const void *g, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(t5_smem_u32(smem)), "l"(g),
                 "r"(bytes)
                 : "memory");
}

// The chunk's products by FP64 FMAs, rows in order: an FMA holds its quadrant's pipe for
// 64 clocks, so what counts is full warps, the same number on every quadrant (the tile's
// outputs in a row over 512 threads); the two shared loads beside it do not matter.
// sym: outputs below the diagonal of L^T R1 are left out (their mirror images are read).
// n = 884736, 96 x 112: 21.0 ms (15.8 with the FMA kernel of k_gram.cu, whose tiles are
// alike: here one CTA of two has 64 columns and one 48); Q^T A Q does half.
template <int NB>
__device__ __noinline__ void xg_fma_chunk(unsigned char *smem, int64_t rbeg, int64_t rend,
                                          const XgOperands &o, int a0, int b0, int BA, int sym,
                                          double *__restrict__ out) {
    constexpr int KT = 32, T = 512, kE = kXgM * NB / T;
    const int kb = o.kb1 + o.kb2, tid = threadIdx.x, W = BA + NB;
    double *t = reinterpret_cast<double *>(smem);            // KT x W
    int *first = reinterpret_cast<int *>(t + KT * (kXgM + NB));  // outputs before row a; their count
    const int na = min(BA, o.ka - a0), nb = min(NB, kb - b0);
    // row a of the tile has the columns from left(a) on
    auto left = [&](int a) { return sym ? max(0, min(min(a0 + a, o.kb1) - b0, nb)) : 0; };
    __syncthreads();
    if (tid == 0) {
        int c = 0;
        for (int a = 0; a < na; ++a) {
            first[a] = c;
            c += nb - left(a);
        }
        first[na] = c;
    }
    __syncthreads();
    const int total = first[na], E = (total + T - 1) / T;
    double acc[kE];
    int at[kE];  // columns of the output's operands in t
#pragma unroll
    for (int e = 0; e < kE; ++e) {
        const int i = tid + e * T;
        acc[e] = 0.0;
        at[e] = BA << 16;
        if (tid < T && i < total) {
            int lo = 0, hi = na;  // first[lo] <= i < first[hi]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (first[mid] <= i)
                    lo = mid;
                else
                    hi = mid;
            }
            at[e] = lo | (BA + left(lo) + i - first[lo]) << 16;
        }
    }
    for (int64_t r0 = rbeg; r0 < rend; r0 += KT) {
        __syncthreads();
        for (int i = tid; i < KT * W; i += kXgThreads) {
            const int r = i / W, c = i % W, b = b0 + c - BA;
            const int64_t row = r0 + r;
            double v = 0.0;
            if (row >= rend) {
            } else if (c < BA) {
                if (a0 + c < o.ka) v = __ldg(o.L + row * o.ldl + a0 + c);
            } else if (b < o.kb1) {
                v = __ldg(o.R1 + row * o.ldr1 + b);
            } else if (b < kb) {
                v = __ldg(o.R2 + row * o.ldr2 + (b - o.kb1));
            }
            t[i] = v;
        }
        __syncthreads();
        if (tid >= T) continue;
        for (int r = 0; r < KT; r += 4) {
            const double *p = t + r * W;
#pragma unroll
            for (int e = 0; e < kE; ++e) {
                if (e >= E) break;
                const double *x = p + (at[e] & 0xffff), *y = p + (at[e] >> 16);
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[e] = fma(x[u * W], y[u * W], acc[e]);
            }
        }
    }
    if (tid >= T) return;
#pragma unroll
    for (int e = 0; e < kE; ++e)
        if (tid + e * T < total) out[(at[e] & 0xffff) * NB + (at[e] >> 16) - BA] = acc[e];
}

// NB = 16 * NC columns of [R1 | R2] per output tile (7 NB <= 512 columns of
// tensor memory); VEC: widths and row strides even and bases 16-byte aligned,
// so a pair of columns is one 16-byte copy.
template <int NC, bool VEC>
__global__ void __launch_bounds__(kXgThreads, 1)
    gram_x64_kernel(int64_t n, int64_t rows_per_chunk, XgOperands o, int BA, int tilesB, int sub,
                    int stages, bool scan, int sym, int line, uint32_t *__restrict__ emax,
                    const unsigned long long *__restrict__ elog, double *__restrict__ part,
                    int *__restrict__ flags, long long polls) {
    constexpr int NB = 16 * NC;
    constexpr int NQ = NB / 4;  // accumulator columns per converter thread
    constexpr unsigned lbo_a = (kXgM / 8) * 128, lbo_b = (kXPlanes * NB / 8) * 128;
    constexpr unsigned b_bytes = (kXgKT / 8) * lbo_b;
    constexpr unsigned buf_bytes = kXgABytes + b_bytes;
    constexpr int tmem_cols = NC == 1 ? 128 : NC == 2 ? 256 : 512;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // [plane buffers x2][raw slots][scales][mbarriers][tmem slot][abort][spread x2]
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform, and known to be
    const int nunits = (BA / 8 + NB / 8) * (kXgKT / 8);
    const int upw = (nunits + kXgConvWarps - 1) / kXgConvWarps;
    double2 *raw = reinterpret_cast<double2 *>(smem_raw + 2 * buf_bytes);
    int *esc = reinterpret_cast<int *>(smem_raw + 2 * buf_bytes +
                                       (size_t)stages * upw * kXgConvWarps * 32 * 16);
    uint64_t *sfull = reinterpret_cast<uint64_t *>(esc + kXgM + NB);
    uint64_t *sfree = sfull + 2;
    uint64_t *gdone = sfree + 2;
    uint64_t *gfree = gdone + 1;
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(gfree + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int tile_a = blockIdx.y / tilesB, tile_b = blockIdx.y % tilesB;
    const int a0 = tile_a * BA, b0 = tile_b * NB;
    const int kb = o.kb1 + o.kb2, kc = o.ka + kb;
    const int64_t rbeg = (int64_t)blockIdx.x * rows_per_chunk;
    const int64_t rend = min(n, rbeg + rows_per_chunk);
    const int64_t nsteps = rend > rbeg ? (rend - rbeg + kXgKT - 1) / kXgKT : 0;
    int *flag = flags + (size_t)blockIdx.x * gridDim.y + blockIdx.y;

    // scales of the tile's columns: from the maxima kernel, or, where the
    // operands stay in L2 (scan), from a pass over the chunk's rows, which leaves them;
    // and the bits by which its elements fall short of them, on average
    int *spread = reinterpret_cast<int *>(tmem_slot + 2);
    if (tid < 2) spread[tid] = 0;
    bool bad = false;
    const bool lined = line != kXgNoLine;
    auto short_bits = [&](uint32_t key, uint64_t logs, uint64_t zeros) {
        if (key == 0u) return 0;  // no element, no error
        const double rows = (double)(rend - rbeg);
        const double d = (rows - (double)zeros) * (double)(((key >> 20) + 1) << 8) - (double)logs +
                         (double)zeros * (kXgSpread << 8);
        return (int)fmin(d / rows + 1.0, 1e6);
    };
    int lacks = 0;
    if (!scan) {
        __syncthreads();  // spread is 0 before anyone's bits go in
        if (tid < BA + NB) {
            const int c = tid < BA ? (a0 + tid < o.ka ? a0 + tid : -1)
                                   : (b0 + tid - BA < kb ? o.ka + b0 + tid - BA : -1);
            uint32_t key = 0u;
            uint64_t logs = 0, zeros = 0;
            if (c >= 0)
                for (int s = 0; s < sub; ++s) {
                    const size_t at = ((size_t)blockIdx.x * sub + s) * kc + c;
                    key = max(key, emax[at]);
                    const uint64_t l = lined ? elog[at] : 0;
                    logs += l & ((1ull << kXgZeroBit) - 1);
                    zeros += l >> kXgZeroBit;
                }
            esc[tid] = x64_scale(key, &bad) << 20;
            if (lined) lacks = short_bits(key, logs, zeros);
        }
    } else {
        uint32_t *keys = reinterpret_cast<uint32_t *>(esc);
        XgLogSum *logs = reinterpret_cast<XgLogSum *>(smem_raw);
        if (tid < BA + NB) {
            keys[tid] = 0u;
            logs[tid] = XgLogSum{0u, 0u, 0u};
        }
        __syncthreads();
        const int tpr = (BA + NB) / 2, rpb = kXgThreads / tpr;
        const int r = tid / tpr, c = 2 * (tid % tpr);
        if (r < rpb) {
            auto col_ptr = [&](int cc, int64_t &ld) -> const double * {
                if (cc < BA) {
                    ld = o.ldl;
                    return a0 + cc < o.ka ? o.L + a0 + cc : nullptr;
                }
                const int g = b0 + cc - BA;
                ld = g < o.kb1 ? o.ldr1 : o.ldr2;
                return g < o.kb1 ? o.R1 + g : g < kb ? o.R2 + (g - o.kb1) : nullptr;
            };
            int64_t l0, l1;
            const double *q0 = col_ptr(c, l0), *q1 = col_ptr(c + 1, l1);
            auto scan_rows = [&](auto with_logs) {
                constexpr bool LOG = decltype(with_logs)::value;
                uint32_t k0 = 0u, k1 = 0u;
                uint64_t s0 = 0, s1 = 0;
                auto take = [&](double x, uint32_t &k, uint64_t &l) {
                    const uint32_t e = x64_key(x);
                    k = max(k, e);
                    if constexpr (LOG) l += xg_log(e);
                };
                if constexpr (VEC) {
                    if (q0) {
#pragma unroll 8
                        for (int64_t row = rbeg + r; row < rend; row += rpb) {
                            const double2 v = __ldg(reinterpret_cast<const double2 *>(q0 + row * l0));
                            take(v.x, k0, s0);
                            take(v.y, k1, s1);
                        }
                    }
                } else {
#pragma unroll 4
                    for (int64_t row = rbeg + r; row < rend; row += rpb) {
                        if (q0) take(__ldg(q0 + row * l0), k0, s0);
                        if (q1) take(__ldg(q1 + row * l1), k1, s1);
                    }
                }
                atomicMax(&keys[c], k0);
                atomicMax(&keys[c + 1], k1);
                if constexpr (LOG) {
                    xg_add(logs[c], s0);
                    xg_add(logs[c + 1], s1);
                }
            };
            if (lined)
                scan_rows(std::true_type());
            else
                scan_rows(std::false_type());
        }
        __syncthreads();
        if (tid < BA + NB) {
            const uint32_t key = keys[tid];
            uint32_t *left = emax + (size_t)blockIdx.x * kc;
            const int c = tid < BA ? a0 + tid : b0 + tid - BA;
            if (tid < BA && tile_b == 0 && c < o.ka) left[c] = key;
            if (tid >= BA && tile_a == 0 && c < kb) left[o.ka + c] = key;
            if (lined) lacks = short_bits(key, xg_logs(logs[tid]), logs[tid].zeros);
            esc[tid] = x64_scale(key, &bad) << 20;
        }
    }
    if (lacks > 0) atomicMax(&spread[tid >= BA], lacks);
    if (__syncthreads_or(bad) || spread[0] + spread[1] > line) {
        xg_fma_chunk<NB>(smem_raw, rbeg, rend, o, a0, b0, BA, sym,
                         part + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * (size_t)BA * NB);
        if (tid == 0) *flag = 0;
        return;
    }

    // (A columns past BA keep whatever shared memory holds: they reach only the
    // accumulator lanes past BA, which nobody reads)
    if (tid == 0) {
        t5_mbar_init(&sfull[0], kXgConvWarps);
        t5_mbar_init(&sfull[1], kXgConvWarps);
        t5_mbar_init(&sfree[0], 1);
        t5_mbar_init(&sfree[1], 1);
        t5_mbar_init(gdone, 1);
        t5_mbar_init(gfree, kXgConvWarps);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         t5_smem_u32(tmem_slot)),
                     "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    t5_fence_proxy_async();
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const unsigned tmem = *tmem_slot;
    auto group_end = [&](int64_t e) { return e % kXgGroup == kXgGroup - 1 || e == nsteps - 1; };

    // outputs of this thread: L column 32 (warp % 4) + lane, tile columns
    // [(warp / 4) NQ, + NQ): sum = ahi 2^24 + alo in units of 2^(Ea + Eb - 2106)
    long long ahi[NQ];
    unsigned alo[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        ahi[q] = 0;
        alo[q] = 0u;
    }
    const int quad = warp & 3, quarter = warp >> 2;

    if (warp < kXgConvWarps) {
        // ------------------------------------------------------ converters
        // unit id = warp + 16 u: column octet id / 4, row octet id % 4; lane:
        // row lane / 4 of the octet, column pair lane % 4
        const int lr = lane >> 2, lc = 2 * (lane & 3);
        const int kg = warp & 3, oct0 = warp >> 2;  // id % 4; id / 4 = oct0 + 4 u
        const int rowt = 8 * kg + lr;
        const int c0 = 8 * oct0 + lc;
        int rleft = (int)(rend - rbeg) - rowt;  // > 0: the next step has this thread's row
        // this thread's row of the next step to copy, at tile column c0
        const double *pL = o.L + (rbeg + rowt) * o.ldl + a0 + c0;
        const double *p1 = o.R1 + (rbeg + rowt) * o.ldr1 + (b0 + c0 - BA);
        const double *p2 = o.R2 + (rbeg + rowt) * o.ldr2 + (b0 + c0 - BA - o.kb1);
        double2 *slot = raw + tid;  // this thread's slots: stage st, unit u at (st upw + u) 512
        auto copy_unit = [&](int st, int u) {
            double2 *dst = slot + (st * upw + u) * (kXgConvWarps * 32);
            const int c = c0 + 32 * u;
            const bool rv = rleft > 0;
            auto src = [&](int e, bool &ok) -> const double * {
                const int col = c + e - BA + b0;
                const double *p = c < BA ? pL : col < o.kb1 ? p1 : p2;
                ok = rv && (c < BA ? a0 + c + e < o.ka : col < kb);
                return ok ? p + 32 * u + e : o.L;
            };
            bool ok;
            const double *s0 = src(0, ok);
            if constexpr (VEC) {
                xg_cp16(dst, s0, ok ? 16 : 0);
            } else {
                xg_cp8(dst, s0, ok ? 8 : 0);
                const double *s1 = src(1, ok);
                xg_cp8(reinterpret_cast<double *>(dst) + 1, s1, ok ? 8 : 0);
            }
        };
        auto next_rows = [&]() {
            rleft -= kXgKT;
            pL += kXgKT * o.ldl;
            p1 += kXgKT * o.ldr1;
            p2 += kXgKT * o.ldr2;
        };
        auto fold = [&](int64_t g) {
            const bool okg = __all_sync(
                0xffffffffu, t5_mbar_wait_or_abort(gdone, (unsigned)(g & 1), abort_flag, polls));
            if (!okg) return false;
            t5_fence_after();
            const unsigned ta = tmem + ((unsigned)(32 * quad) << 16) + (unsigned)(quarter * NQ);
#pragma unroll
            for (int c0 = 0; c0 < NQ; c0 += 4) {
                unsigned r[kXPlanes][4];
#pragma unroll
                for (int d = 0; d < kXPlanes; ++d) t5_ld4_nowait(ta + d * NB + c0, r[d]);
                t5_wait_ld();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    int D[kXPlanes];
#pragma unroll
                    for (int d = 0; d < kXPlanes; ++d) D[d] = __float2int_rn(__uint_as_float(r[d][q]));
                    // |D[d]| <= (d + 1) 2^21: the int products fit
                    const long long h =
                        (long long)(D[0] * 256 + D[1]) * 65536 + (long long)(D[2] * 256 + D[3]);
                    const long long l = (long long)D[4] * 65536 + (long long)D[5] * 256 +
                                        (long long)D[6] + (long long)alo[c0 + q];
                    ahi[c0 + q] += h + (l >> 24);
                    alo[c0 + q] = (unsigned)l & 0xffffffu;
                }
            }
            t5_fence_before();
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(gfree);
            return true;
        };
        for (int st = 0; st < stages; ++st) {
            if (st < nsteps)
                for (int u = 0; u < upw; ++u)
                    if (warp + kXgConvWarps * u < nunits) copy_unit(st, u);
            next_rows();
            t5_cp_commit();
        }
        const int toff = kg * (int)lbo_a + lr * 16 + lc * 2 + oct0 * 128;
        const int boff = (int)kXgABytes + kg * (int)lbo_b + lr * 16 + lc * 2 +
                         (oct0 - BA / 8) * 128;
        bool ok = true;
        int st = 0;
        for (int64_t j = 0; j < nsteps && ok; ++j) {
            const int b = (int)(j & 1);
            if (j >= 2) {
                const bool w =
                    t5_mbar_wait_or_abort(&sfree[b], (unsigned)(((j >> 1) - 1) & 1), abort_flag,
                                          polls);
                if (!__all_sync(0xffffffffu, w)) {
                    ok = false;
                    break;
                }
            }
            // this step's rows have landed; up to stages - 1 later steps are in flight
            switch (stages) {
                case 1: asm volatile("cp.async.wait_group 0;\n" ::: "memory"); break;
                case 2: asm volatile("cp.async.wait_group 1;\n" ::: "memory"); break;
                case 3: asm volatile("cp.async.wait_group 2;\n" ::: "memory"); break;
                default: asm volatile("cp.async.wait_group 3;\n" ::: "memory"); break;
            }
            unsigned char *dbase = smem_raw + b * buf_bytes;
            const bool more = j + stages < nsteps;
#pragma unroll
            for (int u = 0; u < kXgMaxUnits; ++u) {
                if (u >= upw || warp + kXgConvWarps * u >= nunits) break;
                const double2 x = slot[(st * upw + u) * (kXgConvWarps * 32)];
                if (more) copy_unit(st, u);  // into this thread's slot, just read
                const uint2 e = *reinterpret_cast<const uint2 *>(esc + c0 + 32 * u);
                uint32_t w[kXPlanes];
                x64_planes2(x.x, x.y, e.x, e.y, w);
                if (oct0 + 4 * u < BA / 8) {
                    unsigned char *d = dbase + toff + u * 512;
#pragma unroll
                    for (int p = 0; p < kXPlanes; ++p)
                        *reinterpret_cast<uint32_t *>(d + p * (kXgKT / 8) * (int)lbo_a) = w[p];
                } else {
                    unsigned char *d = dbase + boff + u * 512;
#pragma unroll
                    for (int p = 0; p < kXPlanes; ++p)
                        *reinterpret_cast<uint32_t *>(d + p * (NB / 8) * 128) = w[p];
                }
            }
            next_rows();
            if (++st == stages) st = 0;
            t5_cp_commit();
            t5_fence_proxy_async();
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(&sfull[b]);
            if (j >= 1 && group_end(j - 1)) ok = fold((j - 1) / kXgGroup);
        }
        if (ok && nsteps > 0) ok = fold((nsteps - 1) / kXgGroup);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (!ok && lane == 0) *abort_flag = 1;
    } else {
        // ------------- MMA issuer: a whole warp, one elected lane at the MMAs
        int64_t last = -1;
        for (int64_t j = 0; j < nsteps; ++j) {
            const int b = (int)(j & 1);
            const int64_t g = j / kXgGroup;
            const bool w =
                t5_mbar_wait_or_abort(&sfull[b], (unsigned)((j >> 1) & 1), abort_flag, polls) &&
                (j % kXgGroup != 0 || g < 1 ||
                 t5_mbar_wait_or_abort(gfree, (unsigned)((g - 1) & 1), abort_flag, polls));
            if (!__all_sync(0xffffffffu, w)) {
                if (lane == 0) *abort_flag = 1;
                break;
            }
            t5_fence_after();
            const unsigned abase = t5_smem_u32(smem_raw + b * buf_bytes);
            const unsigned bbase = abase + kXgABytes;
            const unsigned tr = (1u << 15) | (1u << 16);  // A, B MN-major
            if (t5_elect()) {
#pragma unroll
                for (int kk = 0; kk < kXgKT / 16; ++kk) {
                    const unsigned first = (j % kXgGroup == 0 && kk == 0) ? 0u : 1u;
#pragma unroll
                    for (int p = 0; p < kXPlanes; ++p) {
                        // plane p of A times planes 0 .. 6 - p of B: accumulators p .. 6
                        const int N = (kXPlanes - p) * NB;
                        const uint64_t ad = t5_desc_lbo(
                            abase + p * (kXgKT / 8) * lbo_a + 2 * kk * lbo_a, lbo_a, 128);
                        const uint64_t bd = t5_desc_lbo(bbase + 2 * kk * lbo_b, lbo_b, 128);
                        const unsigned dt = tmem + p * NB;
                        const unsigned acc = p == 0 ? first : 1u;
                        if (N <= 256) {
                            t5_mma(dt, ad, bd, x64_idesc(kXgM, N) | tr, acc);
                        } else {
                            t5_mma(dt, ad, bd, x64_idesc(kXgM, 256) | tr, acc);
                            const uint64_t bd2 =
                                t5_desc_lbo(bbase + 2 * kk * lbo_b + (256 / 8) * 128, lbo_b, 128);
                            t5_mma(dt + 256, ad, bd2, x64_idesc(kXgM, N > 256 ? N - 256 : 16) | tr, acc);
                        }
                    }
                }
                t5_commit(&sfree[b]);
                if (group_end(j)) t5_commit(gdone);
            }
            __syncwarp();
            last = j;
        }
        // every committed MMA finishes before tensor memory goes (bounded)
        if (last >= 0) {
            t5_mbar_wait(&sfree[last & 1], (unsigned)((last >> 1) & 1));
            if (group_end(last)) t5_mbar_wait(gdone, (unsigned)((last / kXgGroup) & 1));
        }
    }
    t5_fence_before();
    const int gave_up = __syncthreads_or(*abort_flag);
    if (warp == 0) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                     "r"(tmem_cols));
    }
    if (tid == 0) *flag = gave_up;
    if (gave_up || warp >= kXgConvWarps) return;
    const int row_t = 32 * quad + lane;
    if (row_t >= BA) return;
    double *out = part + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * (size_t)BA * NB +
                  (size_t)row_t * NB + quarter * NQ;
    const int ea = (esc[row_t] >> 20) - 2106;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double v = fma((double)ahi[q], 16777216.0, (double)alo[q]);
        out[q] = scalbn(v, ea + (esc[BA + quarter * NQ + q] >> 20));
    }
}

// Sum of the chunks' partials: 16 threads share an output, each sums a
// contiguous sixteenth of the chunks in order, then the sixteenths are added in
// order.  With a raised flag the same threads form the output from L, R1, R2.  The
// blocks from nsum on leave the exponents of L's and R1's columns (eL, eR1) instead.
constexpr int kXrElems = 32, kXrSlices = 16;

__global__ void __launch_bounds__(kXrSlices *kXrElems)
    gram_x64_reduce_kernel(const double *__restrict__ part, int nchunks, int ntiles, int BA, int NB,
                           int tilesB, int64_t n, XgOperands o, double *__restrict__ C1, int ldc1,
                           double *__restrict__ C2, int ldc2, const int *__restrict__ flags,
                           int sym, int nsum, const uint32_t *__restrict__ emax, int groups,
                           int *__restrict__ eL, int *__restrict__ eR1) {
    __shared__ double qs[kXrSlices][kXrElems];
    const int el = threadIdx.x % kXrElems, q = threadIdx.x / kXrElems;
    const int kb = o.kb1 + o.kb2;
    if (blockIdx.x >= nsum) {
        const int c = (blockIdx.x - nsum) * kXrElems + el;
        x64_col_exp(emax, groups, o.ka + kb, c, c < o.ka + (eR1 ? o.kb1 : 0), el, q,
                    reinterpret_cast<float(*)[32]>(qs), c < o.ka ? eL + c : eR1 + (c - o.ka));
        return;
    }
    const int idx = blockIdx.x * kXrElems + el;
    const bool active = idx < o.ka * kb;
    const int a = active ? idx / kb : 0, b = active ? idx % kb : 0;
    double s = 0.0;
    {
        // (sym: below the diagonal of L^T R1, the mirror image)
        const bool lower = sym && b < a && b < o.kb1;
        const int pa = lower ? b : a, pb = lower ? a : b;
        const int tile = (pa / BA) * tilesB + (pb / NB);
        const size_t off = (size_t)tile * BA * NB + (size_t)(pa % BA) * NB + (pb % NB);
        const size_t stride = (size_t)ntiles * BA * NB;
        const int per = (nchunks + kXrSlices - 1) / kXrSlices;
        const int p1 = min(nchunks, q * per + per);
        if (active)
#pragma unroll 10
            for (int p = q * per; p < p1; ++p) s += part[off + (size_t)p * stride];
    }
    int raised = 0;
    for (int i = threadIdx.x; i < nchunks * ntiles; i += blockDim.x) raised |= flags[i];
    if (__syncthreads_or(raised)) {
        s = 0.0;
        if (active) {
            const double *R = b < o.kb1 ? o.R1 + b : o.R2 + (b - o.kb1);
            const int64_t ldr = b < o.kb1 ? o.ldr1 : o.ldr2;
            const int64_t per = (n + kXrSlices - 1) / kXrSlices;
            const int64_t r1 = min(n, q * per + per);
#pragma unroll 8
            for (int64_t r = q * per; r < r1; ++r) s = fma(o.L[r * o.ldl + a], R[r * ldr], s);
        }
    }
    qs[q][el] = s;
    __syncthreads();
    if (q == 0 && active) {
        double t = qs[0][el];
#pragma unroll
        for (int i = 1; i < kXrSlices; ++i) t += qs[i][el];
        if (b < o.kb1)
            C1[(size_t)a * ldc1 + b] = t;
        else
            C2[(size_t)a * ldc2 + (b - o.kb1)] = t;
    }
}

// ------------------------------------------------------------------- host
struct XgPlan {
    int BA, NB, tilesA, tilesB, nchunks, sub, stages;
    bool scan;  // column maxima inside the product kernel
    int64_t rows_per_chunk, rows_per_sub;
    size_t smem, part_bytes, emax_bytes, elog_bytes, total;
};

static XgPlan plan_x64(int64_t n, int ka, int kb) {
    XgPlan p{};
    auto up = [](int64_t x, int64_t q) { return (x + q - 1) / q * q; };
    p.tilesA = (ka + kXgM - 1) / kXgM;
    p.BA = (int)up((ka + p.tilesA - 1) / p.tilesA, 8);
    p.tilesB = (kb + 63) / 64;
    p.NB = (int)up((kb + p.tilesB - 1) / p.tilesB, 16);
    const int tiles = p.tilesA * p.tilesB;
    // one CTA per SM in all; chunks of at least two steps
    int64_t nch = std::max<int64_t>(1, sm_count() / tiles);
    p.rows_per_chunk = std::max<int64_t>(up((n + nch - 1) / nch, kXgKT), 2 * kXgKT);
    p.nchunks = (int)std::max<int64_t>(1, (n + p.rows_per_chunk - 1) / p.rows_per_chunk);
    const int64_t sub = std::max<int64_t>(
        1, std::min<int64_t>(std::min<int64_t>(8, 1024 / p.nchunks), p.rows_per_chunk / 128));
    p.rows_per_sub = up((p.rows_per_chunk + sub - 1) / sub, 8);
    p.sub = (int)((p.rows_per_chunk + p.rows_per_sub - 1) / p.rows_per_sub);
    const int nunits = (p.BA / 8 + p.NB / 8) * (kXgKT / 8);
    const int upw = (nunits + kXgConvWarps - 1) / kXgConvWarps;
    const size_t planes = 2 * ((size_t)kXgABytes + (size_t)(kXgKT / 8) * (kXPlanes * p.NB / 8) * 128);
    const size_t tables = (size_t)(kXgM + p.NB) * 4 + 6 * 8 + 16;
    const size_t stage = (size_t)upw * kXgConvWarps * 32 * 16;
    // raw steps in flight: with few columns a step's work is shorter than the
    // latency of its copies
    p.stages = kXgMaxStages;
    while (p.stages > 1 && planes + tables + p.stages * stage > max_smem_optin()) --p.stages;
    p.smem = planes + tables + p.stages * stage;
    // small operands are read twice by the product kernel, which saves a launch
    // (n = 16384, k = 4 (+1): 22.1 us with the maxima kernel, 20.4 without; n = 50653,
    // k = 20 (+5): 41.7 either way); larger ones by a maxima kernel on more blocks
    p.scan = (double)n * (ka * p.tilesB + (double)kb * p.tilesA) * 8.0 <= 4e6;
    p.part_bytes = (size_t)p.nchunks * tiles * p.BA * p.NB * sizeof(double);
    p.elog_bytes = (size_t)p.nchunks * p.sub * (ka + kb) * 8;
    p.emax_bytes = p.elog_bytes / 2;
    p.total = p.part_bytes + p.elog_bytes + p.emax_bytes + (size_t)p.nchunks * tiles * sizeof(int) + 64;
    return p;
}

size_t gram_x64_workspace_bytes(int64_t n, int ka, int kb) {
    size_t b = 0;  // any narrower product with the same workspace fits as well
    for (int w = 16; w < kb; w += 16) b = std::max(b, plan_x64(n, ka, w).total);
    return std::max(b, plan_x64(n, ka, kb).total);
}

// n < 256: an FMA chain of so few rows rounds less than the planes drop.  Above, for
// the columns that gram_tiny_kernel leaves, this kernel is the faster one but for a
// tie at the fewest: through cacg_k_gram (some 15 us of it the call), planes and FMAs,
// n = 1369 / 16384 / 884736: 20 x 25 26 / 38 / 383 us against 24 / 39 / 870; 32 x 40
// 30 / 40 / 414 against 37 / 63 / 1975; 96 x 112 42 / 69 / 1088 against 194 / 382 / 15816.
bool gram_x64_supported(int64_t n, int ka, int kb) {
    return n >= 256 && ka > 0 && kb > 0 && ka <= 256 && kb <= 512;
}

template <int NC, bool VEC>
static void xg_launch(dim3 grid, const XgPlan &p, cudaStream_t st, int64_t n, const XgOperands &o,
                      int sym, int line, uint32_t *emax, const unsigned long long *elog, double *part,
                      int *flags) {
    set_smem_attr(gram_x64_kernel<NC, VEC>, (int)max_smem_optin());
    gram_x64_kernel<NC, VEC><<<grid, kXgThreads, p.smem, st>>>(
        n, p.rows_per_chunk, o, p.BA, p.tilesB, p.sub, p.stages, p.scan, sym, line, emax, elog, part, flags,
        pipeline_wait_limit());
}

int launch_gram_x64(cudaStream_t st, int64_t n, const double *L, int64_t ldl, int ka,
                    const double *R1, int64_t ldr1, int kb1, const double *R2, int64_t ldr2,
                    int kb2, double *C1, int ldc1, double *C2, int ldc2, double *ws,
                    size_t ws_bytes, bool symmetric, bool normwise, ColExps *ce) {
    const int kb = kb1 + kb2;
    if (!gram_x64_supported(n, ka, kb)) return CACG_ERR_UNSUPPORTED;
    const XgPlan p = plan_x64(n, ka, kb);
    if (p.total > ws_bytes || !ws || p.smem > max_smem_optin()) return CACG_ERR_UNSUPPORTED;
    double *part = ws;
    unsigned long long *elog =
        reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(ws) + p.part_bytes);
    uint32_t *emax = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(elog) + p.elog_bytes);
    int *flags = reinterpret_cast<int *>(reinterpret_cast<char *>(emax) + (p.emax_bytes + 15) / 16 * 16);
    const XgOperands o{L, R1, R2, ldl, ldr1, ldr2, ka, kb1, kb2};
    const int sym = symmetric && ka == kb1;
    const int line = normwise ? kXgNoLine : kXgSpread << 8;
    // 16-byte pairs: even widths, even strides, aligned bases
    const bool vec = ka % 2 == 0 && kb1 % 2 == 0 && kb2 % 2 == 0 && ldl % 2 == 0 &&
                     ldr1 % 2 == 0 && aligned16(L) && aligned16(R1) &&
                     (kb2 == 0 || (ldr2 % 2 == 0 && aligned16(R2)));
    const dim3 mgrid(p.nchunks, p.sub);
    int rc = CACG_OK;
    if (p.scan) {
    } else {
        auto kernel = vec ? (normwise ? gram_x64_colmax_kernel<true, false>
                                      : gram_x64_colmax_kernel<true, true>)
                          : (normwise ? gram_x64_colmax_kernel<false, false>
                                      : gram_x64_colmax_kernel<false, true>);
        kernel<<<mgrid, 512, 0, st>>>(n, p.rows_per_chunk, p.rows_per_sub, o, emax, elog);
    }
    if (!p.scan) rc = check_launch();
    if (rc != CACG_OK) return rc;
    const dim3 grid(p.nchunks, p.tilesA * p.tilesB);
#define XG_CASE(NC)                                                       \
    case NC:                                                              \
        if (vec)                                                          \
            xg_launch<NC, true>(grid, p, st, n, o, sym, line, emax, elog, part, flags);    \
        else                                                              \
            xg_launch<NC, false>(grid, p, st, n, o, sym, line, emax, elog, part, flags);   \
        break;
    switch (p.NB / 16) {
        XG_CASE(1)
        XG_CASE(2)
        XG_CASE(3)
        XG_CASE(4)
        default:
            return CACG_ERR_UNSUPPORTED;
    }
#undef XG_CASE
    rc = check_launch();
    if (rc != CACG_OK) return rc;
    const int nsum = (ka * kb + kXrElems - 1) / kXrElems;
    const int nexp = ce ? (ka + (ce->R1 ? kb1 : 0) + kXrElems - 1) / kXrElems : 0;
    gram_x64_reduce_kernel<<<nsum + nexp, kXrSlices * kXrElems, 0, st>>>(
        part, p.nchunks, p.tilesA * p.tilesB, p.BA, p.NB, p.tilesB, n, o, C1, ldc1, C2, ldc2, flags, sym,
        nsum, emax, p.nchunks * (p.scan ? 1 : p.sub), ce ? ce->L : nullptr, ce ? ce->R1 : nullptr);
    if (ce) ce->set = true;
    return check_launch();
}

__global__ void __launch_bounds__(kXrSlices *kXrElems)
    col_exps_kernel(const uint32_t *__restrict__ emax, int groups, int k, int kc,
                    int *__restrict__ e0, int *__restrict__ e1) {
    __shared__ float sh[kXrSlices][kXrElems];
    const int el = threadIdx.x % kXrElems, q = threadIdx.x / kXrElems;
    const int c = blockIdx.x * kXrElems + el;
    x64_col_exp(emax, groups, kc, c, c < kc, el, q, sh, c < k ? e0 + c : e1 + (c - k));
}

int launch_col_exps(cudaStream_t st, int64_t n, int k, const double *A0, const double *A1,
                    int64_t lda, double *ws, size_t ws_bytes, int *e0, int *e1) {
    if (n <= 0 || k <= 0 || k > 256) return CACG_ERR_UNSUPPORTED;
    const int kc = A1 ? 2 * k : k;
    const int64_t rows = std::max<int64_t>(64, (n + 2 * sm_count() - 1) / (2 * sm_count()));
    const int groups = (int)((n + rows - 1) / rows);
    if (!ws || (size_t)groups * kc * 4 > ws_bytes) return CACG_ERR_UNSUPPORTED;
    uint32_t *emax = reinterpret_cast<uint32_t *>(ws);
    const XgOperands o{A0, A1, nullptr, lda, lda, 0, k, A1 ? k : 0, 0};
    if (k % 2 == 0 && lda % 2 == 0 && aligned16(A0) && (!A1 || aligned16(A1)))
        gram_x64_colmax_kernel<true, false><<<dim3(groups, 1), 512, 0, st>>>(n, rows, rows, o, emax, nullptr);
    else
        gram_x64_colmax_kernel<false, false><<<dim3(groups, 1), 512, 0, st>>>(n, rows, rows, o, emax, nullptr);
    int rc = check_launch();
    if (rc != CACG_OK) return rc;
    col_exps_kernel<<<(kc + kXrElems - 1) / kXrElems, kXrSlices * kXrElems, 0, st>>>(emax, groups, k, kc,
                                                                                   e0, e1);
    return check_launch();
}

}  // namespace cacg
