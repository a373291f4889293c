// k_dia_fix.cu -- FP64 SpMM over the DIA view of matrices whose off-diagonal
// nonzeros all have one value (finite-difference stencils with constant
// coefficients; the main diagonal is arbitrary), with the neighbour sums in
// 64-bit fixed point.
//
// Reference operations replaced (sclc/cacg): as k_dia.cu (spmm_csr_v1
// src/BLAS3.c:20-155, spmm_csr_info_data_sep_BCBCG src/BLAS3.c:913-976 and the
// basis axpbys src/BLAS3.c:828-847, 978-994), in FP64.
//
// Why: the FP64 pipe does 2 FMAs a clock per SM, so a 27-point row costs 13
// clocks a column there, the integer pipe's additions 1.  With c the common
// off-diagonal value, A x = D x + c sum_j x_j: x is written once as 57-bit
// integers on a scale per column, the sum over the neighbours present in a row
// (a bit per diagonal) is exact, and the FP64 pipe is left with one conversion
// and two FMAs per output:
//     Y = ca c S + (ca D [+ cb]) X + cb Z1 + cc Z2      (cb folded in if Z1 is X)
// Each x is rounded at 2^-58 of its column's largest element M, once; the FMA chain
// rounds at 2^-53 of every partial sum.  For spread columns that is the smaller
// error: per row the roundings of d neighbours leave 2^-59.8 sqrt(d) M |c|, the FMAs'
// (random signs) about 2^-54.3 sqrt(d (d + 1) / 2) rms(x) |c|, which is more while
// M < 45 rms (5 and 7 points; 84 at 27).  So a column needs an eighth of its elements
// at M / 16 or above (then M <= 45 rms; normal data has 62 %, a solver's basis more):
// where one has not, a point source say, the product takes FP64 FMAs.
//
// Measured at 27 points, n = 262144, w = 16 (75 us a step): FP64 pipe 62 % busy,
// the rest the latency of the window reads; four rows a thread and three CTAs an
// SM beat eight rows and two (91 us).  The sums are normalised to FP64 by integer
// instructions, which leaves the FP64 pipe half as busy (35 -> 31 us a 7-point
// step, n = 262144, w = 8).
//
// Three launches: column maxima (partials per block; left out in a chain of
// basis steps, where the step that wrote X has left them), conversion (which
// first reduces them, and counts the large elements), and the product.  A column with
// Inf or NaN, or whose results could leave FP64's normal numbers by the exponent
// additions, sends the product to the FMAs too: over the DIA values, with the same
// windows, at the FP64 pipe's rate.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "cacg_internal.cuh"
#include "cacg_solver.h"
#include "x64_util.cuh"

namespace cacg {

namespace {

constexpr int kFixThreads = 256;
constexpr int kFixR = 4;                       // rows per thread
constexpr int kFixW = kFixR + kDiaGroupMax - 1;  // window rows
constexpr int kFixMaxBlocks = 608;             // partial maxima per column

// mask[row]: bit d set where diagonal d of the row holds c, 0 in rows [npad, nall);
// *bad when an off-diagonal value is neither 0 nor c
__global__ void fix_mask_kernel(int64_t npad, int64_t nall, DiaDesc desc, int dmain,
                                const double *__restrict__ v64, double c,
                                uint32_t *__restrict__ mask, int *__restrict__ bad) {
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < nall;
         row += (int64_t)gridDim.x * blockDim.x) {
        uint32_t m = 0u;
        bool ok = true;
        for (int d = 0; row < npad && d < desc.ndiag; ++d) {
            if (d == dmain) continue;
            const double v = v64[(size_t)d * npad + row];
            if (v == c)
                m |= 1u << d;
            else if (v != 0.0)
                ok = false;
        }
        mask[row] = m;
        if (!ok) atomicOr(bad, 1);
    }
}

// part[block * w + column]
template <bool VEC>
__global__ void __launch_bounds__(kFixThreads)
    fix_colmax_kernel(int64_t n, int w, const double *__restrict__ X, int64_t ldx,
                      uint32_t *__restrict__ part, uint32_t *__restrict__ large) {
    extern __shared__ uint32_t fix_mx[];
    for (int i = threadIdx.x; i < w; i += blockDim.x) {
        fix_mx[i] = 0u;
        if (blockIdx.x == 0) large[i] = 0u;  // the conversion's counters
    }
    __syncthreads();
    const int tpr = VEC ? w / 2 : w;
    const int rpb = blockDim.x / tpr;
    const int r = threadIdx.x / tpr, c = (threadIdx.x % tpr) * (VEC ? 2 : 1);
    if (r < rpb) {
        uint32_t k0 = 0u, k1 = 0u;
#pragma unroll 4
        for (int64_t row = (int64_t)blockIdx.x * rpb + r; row < n; row += (int64_t)gridDim.x * rpb) {
            if constexpr (VEC) {
                const double2 v = __ldg(reinterpret_cast<const double2 *>(X + row * ldx + c));
                k0 = max(k0, x64_key(v.x));
                k1 = max(k1, x64_key(v.y));
            } else {
                k0 = max(k0, x64_key(__ldg(X + row * ldx + c)));
            }
        }
        atomicMax(&fix_mx[c], k0);
        if constexpr (VEC) atomicMax(&fix_mx[c + 1], k1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < w; i += blockDim.x) part[(size_t)blockIdx.x * w + i] = fix_mx[i];
}

// round(x 2^(1079 - E)), |x| < 2^(E - 1022): |result| <= 2^57
__device__ __forceinline__ long long fix_from(double x, int E) {
    const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
    const int s = E - (int)((xh >> 20) & 0x7ffu);
    const uint32_t mh = (xh & 0xfffffu) | 0x100000u;
    const uint64_t m5 = ((uint64_t)__funnelshift_l(xl, mh, 5) << 32) | (uint64_t)(xl << 5);
    uint64_t m;  // twice the magnitude
    asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m5), "r"(s));
    const long long a = (long long)((m + 1) >> 1);
    return (int32_t)xh < 0 ? -a : a;
}

// a column's scale exponent from its largest key; *bad beyond 2^+-range (Inf and NaN too)
__device__ __forceinline__ int fix_scale(uint32_t key, int range, bool *bad) {
    const int e = (int)(key >> 20);
    if (key != 0u && (e < 1023 - range || e > 1023 + range)) *bad = true;
    return key == 0u ? 1023 : e;
}

// an element of M / 16 or above (M: the power of two above its column's largest),
// and every one of a zero column
__device__ __forceinline__ uint32_t fix_large(double x, int E, int within) {
    return E - (int)(((uint32_t)__double2hiint(x) >> 20) & 0x7ffu) <= within ? 1u : 0u;
}

// xi (n x wp, wp = w rounded up to even, the padding column zero); scale[0 .. w):
// the columns' exponents, scale[w]: raised when a column has none; large[0 .. w):
// counts of large elements, added up over the blocks
template <bool VEC>
__global__ void __launch_bounds__(kFixThreads)
    fix_convert_kernel(int64_t n, int w, int wp, const double *__restrict__ X, int64_t ldx,
                       const uint32_t *__restrict__ part, int nparts, int range,
                       long long *__restrict__ xi, int *__restrict__ scale,
                       uint32_t *__restrict__ large) {
    extern __shared__ uint32_t fix_mx[];
    uint32_t *cnt = fix_mx + wp;
    for (int i = threadIdx.x; i < 2 * wp; i += blockDim.x) fix_mx[i] = 0u;
    __syncthreads();
    // stripes of the partials: one atomic per thread and column group
    const int ns = max(1, (int)blockDim.x / w);
    if (threadIdx.x < ns * w || w > (int)blockDim.x) {
        for (int c = threadIdx.x % w; c < w; c += blockDim.x) {
            uint32_t k = 0u;
#pragma unroll 8
            for (int p = threadIdx.x / w; p < nparts; p += ns) k = max(k, part[(size_t)p * w + c]);
            atomicMax(&fix_mx[c], k);
        }
    }
    __syncthreads();
    bool bad = false;
    for (int i = threadIdx.x; i < wp; i += blockDim.x) {
        const uint32_t key = fix_mx[i];
        const int e = fix_scale(key, range, &bad);
        fix_mx[i] = (uint32_t)e;
        cnt[i] = key == 0u ? 0x80000000u : 0u;  // the top bit: a zero column
        if (blockIdx.x == 0 && i < w) scale[i] = e;
    }
    const int any = __syncthreads_or(bad);
    if (blockIdx.x == 0 && threadIdx.x == 0) scale[w] = any;
    if (any) return;
    const int tpr = wp / 2;
    const int rpb = blockDim.x / tpr;
    const int r = threadIdx.x / tpr, c = (threadIdx.x % tpr) * 2;
    const bool on = r < rpb;
    const int e0 = on ? (int)fix_mx[c] : 0, e1 = on ? (int)fix_mx[c + 1] : 0;
    const int in0 = on && cnt[c] ? INT32_MAX : 3, in1 = on && cnt[c + 1] ? INT32_MAX : 3;
    uint32_t n0 = 0u, n1 = 0u;
#pragma unroll 4
    for (int64_t row = (int64_t)blockIdx.x * rpb + r; on && row < n;
         row += (int64_t)gridDim.x * rpb) {
        double2 v = make_double2(0.0, 0.0);
        if constexpr (VEC) {
            v = __ldg(reinterpret_cast<const double2 *>(X + row * ldx + c));
        } else {
            v.x = __ldg(X + row * ldx + c);
            if (c + 1 < w) v.y = __ldg(X + row * ldx + c + 1);
        }
        *reinterpret_cast<longlong2 *>(xi + row * wp + c) =
            make_longlong2(fix_from(v.x, e0), fix_from(v.y, e1));
        n0 += fix_large(v.x, e0, in0);
        n1 += fix_large(v.y, e1, in1);
    }
    __syncthreads();  // every thread has seen the zero columns' bits
    if (on) {
        atomicAdd(&cnt[c], n0);
        atomicAdd(&cnt[c + 1], n1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < w; i += blockDim.x)
        atomicAdd(&large[i], cnt[i] & 0x7fffffffu);
}

struct FixArgs {
    int64_t n, npad;
    int w, wp, cpr, runs;  // columns; 2-column chunks a row; row runs per block
    const uint32_t *mask;
    const double *vals;  // DIA values (npad apart); the main diagonal is diagonal dmain
    int dmain;           // -1: no main diagonal
    double c, ca, cb, cc;
    int c_pow2;  // ca c = +-2^c_pow2 (0 when it is no power of two)
    int fold;    // Z1 is X: cb goes into the diagonal's factor
    const double *X, *Z1, *Z2;
    int64_t ldx, ldz1, ldz2, ldy;
    double *Y;
    const long long *xi;
    const int *scale;
    const uint32_t *large;
    uint32_t *ymax;   // column maxima of Y, a partial per block (NULL: not wanted) ...
    uint32_t *large0;  // ... and the counters of the call that takes Y, zeroed here
};

template <bool VEC>
__device__ __forceinline__ double2 fix_ld(const double *p, int c, int w) {
    if constexpr (VEC) {
        return *reinterpret_cast<const double2 *>(p + c);
    } else {
        return make_double2(p[c], c + 1 < w ? p[c + 1] : 0.0);
    }
}

// VEC: even w and strides, 16-byte aligned X, Y, Z1, Z2
// MODE: the addends besides the diagonal's, by FP64 operations per output (half
// of one for the diagonal's factor):
//   kFixPow2  none, ca c = +-2^c_pow2 (one FMA)
//   kFixNone  none (two);  kFixStep  Z2 with cc = -1 (two);  kFixAny  (up to four)
enum { kFixPow2 = 0, kFixNone = 1, kFixStep = 2, kFixAny = 3 };

template <bool VEC, int MODE>
__global__ void __launch_bounds__(kFixThreads, 3)
    fix_spmm_kernel(const __grid_constant__ FixArgs a, const __grid_constant__ DiaDesc desc) {
    extern __shared__ uint32_t fix_mx[];
    const int lr = threadIdx.x / a.cpr, c = 2 * (threadIdx.x % a.cpr);
    const int BR = a.runs * kFixR;
    const int64_t nblk = lr < a.runs ? (a.n + BR - 1) / BR : 0;
    uint32_t k0 = 0u, k1 = 0u;
    auto put_max = [&]() {
        if (!a.ymax) return;
        for (int i = threadIdx.x; i < a.wp; i += blockDim.x) fix_mx[i] = 0u;
        __syncthreads();
        if (lr < a.runs) {
            atomicMax(&fix_mx[c], k0);
            atomicMax(&fix_mx[c + 1], k1);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < a.w; i += blockDim.x)
            a.ymax[(size_t)blockIdx.x * a.w + i] = fix_mx[i];
    };
    bool spread = a.scale[a.w] == 0;
    for (int i = threadIdx.x; i < a.w; i += blockDim.x) {
        spread = spread && (int64_t)a.large[i] * 8 >= a.n;
        if (a.ymax && blockIdx.x == 0) a.large0[i] = 0u;
    }
    const bool fixed = __syncthreads_and(spread) != 0;
    const int e0 = c < a.w ? a.scale[c] : 1023, e1 = c + 1 < a.w ? a.scale[c + 1] : 1023;
    const double cac = a.ca * a.c;
    const int flip = cac < 0.0 ? (int)0x80000000 : 0;
    // ca c on the columns' scales
    const double c0 = scalbn(cac, e0 - 1079), c1 = scalbn(cac, e1 - 1079);
    const double fca = a.ca, fcb = a.fold ? a.cb : 0.0;
    // FIXED: sums of xi over the presence bits; else FMAs of X over the DIA values
    auto rows = [&](auto mode) {
        constexpr bool FIXED = decltype(mode)::value;
        using P = typename std::conditional<FIXED, longlong2, double2>::type;
        for (int64_t blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
            const int64_t r0 = blk * BR + (int64_t)lr * kFixR;
            uint32_t m[kFixR];
            if constexpr (FIXED) {
                const uint4 m0 = __ldg(reinterpret_cast<const uint4 *>(a.mask + r0));
                m[0] = m0.x, m[1] = m0.y, m[2] = m0.z, m[3] = m0.w;
            }
            P acc[kFixR];
#pragma unroll
            for (int i = 0; i < kFixR; ++i) acc[i].x = acc[i].y = 0;
            for (int g = 0; g < desc.ngroups; ++g) {
                const int d0 = desc.gstart[g], G = desc.gstart[g + 1] - d0;
                const int64_t x0 = r0 + desc.off[d0];
                P win[kFixW];
                if constexpr (FIXED) {
                    if (x0 >= 0 && x0 + kFixW <= a.n) {
                        const long long *xp = a.xi + x0 * a.wp + c;
#pragma unroll
                        for (int t = 0; t < kFixW; ++t)
                            if (t < kFixR + G - 1)
                                win[t] =
                                    __ldg(reinterpret_cast<const longlong2 *>(xp + (int64_t)t * a.wp));
                    } else {
#pragma unroll
                        for (int t = 0; t < kFixW; ++t) {
                            if (t < kFixR + G - 1) {
                                int64_t xr = x0 + t;
                                xr = xr < 0 ? 0 : (xr >= a.n ? a.n - 1 : xr);  // its bit is clear
                                win[t] = __ldg(
                                    reinterpret_cast<const longlong2 *>(a.xi + xr * a.wp + c));
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < kFixW; ++t) {
                        if (t < kFixR + G - 1) {
                            const int64_t xr = x0 + t;
                            win[t] = make_double2(0.0, 0.0);
                            if (xr >= 0 && xr < a.n) win[t] = fix_ld<VEC>(a.X + xr * a.ldx, c, a.w);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < kDiaGroupMax; ++j) {
                    if (j < G) {
                        if constexpr (FIXED) {
                            const uint32_t bit = 1u << (d0 + j);
#pragma unroll
                            for (int i = 0; i < kFixR; ++i) {
                                if (m[i] & bit) {
                                    acc[i].x += win[i + j].x;
                                    acc[i].y += win[i + j].y;
                                }
                            }
                        } else {
                            // (rows past n: zeros up to npad, the presence words behind it)
                            const double *vp = a.vals + (size_t)(d0 + j) * a.npad + r0;
#pragma unroll
                            for (int i = 0; i < kFixR; ++i) {
                                const double v = r0 + i < a.n ? __ldg(vp + i) : 0.0;
                                acc[i].x = fma(v, win[i + j].x, acc[i].x);
                                acc[i].y = fma(v, win[i + j].y, acc[i].y);
                            }
                        }
                    }
                }
            }
            const double *dv = a.dmain >= 0 ? a.vals + (size_t)a.dmain * a.npad + r0 : nullptr;
#pragma unroll
            for (int i = 0; i < kFixR; ++i) {
                const int64_t row = r0 + i;
                if (row >= a.n) break;
                double2 y;
                if constexpr (!FIXED) {
                    y = make_double2(a.ca * acc[i].x, a.ca * acc[i].y);
                    if (a.Z1) {
                        const double2 z = fix_ld<VEC>(a.Z1 + row * a.ldz1, c, a.w);
                        y.x = fma(a.cb, z.x, y.x);
                        y.y = fma(a.cb, z.y, y.y);
                    }
                    if (a.Z2) {
                        const double2 z = fix_ld<VEC>(a.Z2 + row * a.ldz2, c, a.w);
                        y.x = fma(a.cc, z.x, y.x);
                        y.y = fma(a.cc, z.y, y.y);
                    }
                } else {
                    const double f = fma(fca, dv ? __ldg(dv + i) : 0.0, fcb);
                    const double2 x = fix_ld<VEC>(a.X + row * a.ldx, c, a.w);
                    double t0 = x64_from_ll(acc[i].x), t1 = x64_from_ll(acc[i].y);
                    if constexpr (MODE == kFixPow2) {
                        // the scale, ca c and its sign go into the exponent field
                        t0 = x64_scaled(t0, acc[i].x == 0, e0 - 1079 + a.c_pow2);
                        t1 = x64_scaled(t1, acc[i].y == 0, e1 - 1079 + a.c_pow2);
                        t0 = __hiloint2double(__double2hiint(t0) ^ flip, __double2loint(t0));
                        t1 = __hiloint2double(__double2hiint(t1) ^ flip, __double2loint(t1));
                        y = make_double2(fma(f, x.x, t0), fma(f, x.y, t1));
                    } else {
                        if constexpr (MODE == kFixStep) {
                            const double2 z = fix_ld<VEC>(a.Z2 + row * a.ldz2, c, a.w);
                            y = make_double2(fma(f, x.x, -z.x), fma(f, x.y, -z.y));
                        } else {
                            y = make_double2(f * x.x, f * x.y);
                        }
                        y.x = fma(t0, c0, y.x);
                        y.y = fma(t1, c1, y.y);
                        if constexpr (MODE == kFixAny) {
                            if (a.Z1 && !a.fold) {
                                const double2 z = fix_ld<VEC>(a.Z1 + row * a.ldz1, c, a.w);
                                y.x = fma(a.cb, z.x, y.x);
                                y.y = fma(a.cb, z.y, y.y);
                            }
                            if (a.Z2) {
                                const double2 z = fix_ld<VEC>(a.Z2 + row * a.ldz2, c, a.w);
                                y.x = fma(a.cc, z.x, y.x);
                                y.y = fma(a.cc, z.y, y.y);
                            }
                        }
                    }
                }
                k0 = max(k0, x64_key(y.x));
                k1 = max(k1, x64_key(y.y));
                double *yp = a.Y + row * a.ldy + c;
                if constexpr (VEC) {
                    *reinterpret_cast<double2 *>(yp) = y;
                } else {
                    yp[0] = y.x;
                    if (c + 1 < a.w) yp[1] = y.y;
                }
            }
        }
    };
    if (fixed)
        rows(std::true_type());
    else
        rows(std::false_type());
    put_max();
}

}  // namespace

// The one-value view is worth a look: the first off-diagonal nonzero, finite and of
// moderate size, is every other's value in 64 rows spread over the matrix.
bool dia_fix_candidate(const cacg_csr *A, double *c) {
    double cv = 0.0;
    bool found = false;
    for (int64_t i = 0; i < A->n && !found; ++i)
        for (int32_t e = A->row_ptr[i]; e < A->row_ptr[i + 1]; ++e)
            if (A->col_idx[e] != i && A->val[e] != 0.0) {
                cv = A->val[e];
                found = true;
                break;
            }
    if (!found || !std::isfinite(cv) || std::fabs(cv) < 1e-200 || std::fabs(cv) > 1e200)
        return false;
    for (int t = 0; t < 64; ++t) {
        const int64_t i = A->n / 64 * t + A->n % 64 * t / 64;
        for (int32_t e = A->row_ptr[i]; e < A->row_ptr[i + 1]; ++e)
            if (A->col_idx[e] != i && A->val[e] != 0.0 && A->val[e] != cv) return false;
    }
    *c = cv;
    return true;
}

// presence words behind v64's values, and the padding the kernels read past npad;
// *bad (0 before) set when an off-diagonal value is neither 0 nor c
int launch_dia_fix_mask(cudaStream_t st, int64_t npad, const DiaDesc &desc, double *v64, double c,
                        uint32_t **mask, int *dmain, int *bad) {
    const int64_t nall = npad + kFixThreads * kFixR;
    *mask = reinterpret_cast<uint32_t *>(v64 + (size_t)desc.ndiag * npad);
    *dmain = -1;
    for (int d = 0; d < desc.ndiag; ++d)
        if (desc.off[d] == 0) *dmain = d;
    const int blocks = (int)std::min<int64_t>((nall + 255) / 256, (int64_t)sm_count() * 16);
    fix_mask_kernel<<<blocks, 256, 0, st>>>(npad, nall, desc, *dmain, v64, c, *mask, bad);
    return check_launch();
}

size_t dia_fix_scratch_bytes(int64_t n, int w) {
    const size_t wp = (size_t)(w + 1) / 2 * 2;
    return (size_t)n * wp * 8;
}
size_t dia_fix_mask_bytes(int64_t npad) {
    return (size_t)(npad + kFixThreads * kFixR) * 4 + 16;
}
size_t dia_fix_small_bytes(int w) { return ((size_t)2 * kFixMaxBlocks * w + 3 * w + 1) * 4; }

int launch_dia_fix(cudaStream_t st, const DevMatrix *A, int w, const double *X, int64_t ldx,
                   double *Y, int64_t ldy, const double *Z1, int64_t ldz1, const double *Z2,
                   int64_t ldz2, double ca, double cb, double cc, void *xi, void *small, FixChain *chain) {
    if (!A->fix_mask || !xi || !small || w <= 0 || w > 2 * kFixThreads) return CACG_ERR_UNSUPPORTED;
    if ((double)A->nnz * w < kDiaFixMin) return CACG_ERR_UNSUPPORTED;
    const double cac = ca * A->fix_c;
    if (!std::isfinite(cac)) return CACG_ERR_UNSUPPORTED;
    FixArgs a{};
    a.n = A->n;
    a.npad = A->dia_npad;
    a.w = w;
    a.wp = (w + 1) / 2 * 2;
    a.cpr = a.wp / 2;
    a.runs = std::max(1, std::min(kFixThreads / a.cpr, 128));
    a.mask = A->fix_mask;
    a.vals = A->dia64;
    a.dmain = A->fix_dmain;
    a.c = A->fix_c;
    a.ca = ca, a.cb = cb, a.cc = cc;
    int ex = 0;
    const double fr = std::frexp(std::fabs(cac), &ex);  // 0.5 for a power of two
    // results by exponent additions or by a scaled ca c: normal numbers for columns
    // within 2^+-range
    const bool pow2 = fr == 0.5 && ex > -300 && ex < 300;
    const int range = ex > -100 && ex < 100 ? 800 : 400;
    a.c_pow2 = pow2 ? ex - 1 : 0;
    a.fold = Z1 && Z1 == X && ldz1 == ldx;
    a.X = X, a.Z1 = Z1, a.Z2 = Z2, a.Y = Y;
    a.ldx = ldx, a.ldz1 = ldz1, a.ldz2 = ldz2, a.ldy = ldy;
    a.xi = (const long long *)xi;
    uint32_t *parts = (uint32_t *)small;  // two sets: of X, and of Y for the next step
    int *scale = (int *)(parts + (size_t)2 * kFixMaxBlocks * w);
    uint32_t *larges = (uint32_t *)scale + w + 1;  // two sets as well
    const bool known = chain && chain->of == X && chain->w == w;
    uint32_t *large = larges + (size_t)(known ? chain->set : 0) * w;
    a.large = large;
    uint32_t *part = parts + (size_t)(known ? chain->set : 0) * kFixMaxBlocks * w;
    a.scale = scale;
    const bool xvec = w % 2 == 0 && ldx % 2 == 0 && aligned16(X);
    const bool vec = xvec && ldy % 2 == 0 && aligned16(Y) &&
                     (!Z1 || (ldz1 % 2 == 0 && aligned16(Z1))) &&
                     (!Z2 || (ldz2 % 2 == 0 && aligned16(Z2)));
    const int tpr = xvec ? w / 2 : w;
    const int rpb = kFixThreads / tpr > 0 ? kFixThreads / tpr : 1;
    if (tpr > kFixThreads) return CACG_ERR_UNSUPPORTED;
    int g1 = (int)std::max<int64_t>(
        1, std::min<int64_t>(std::min<int64_t>(kFixMaxBlocks, 4 * (int64_t)sm_count()),
                             (A->n + 4 * rpb - 1) / (4 * rpb)));
    const size_t sm = (size_t)2 * (w + 2) * 4;
    int rc = CACG_OK;
    if (known)
        g1 = chain->nparts;  // the step that wrote X left its maxima
    else if (xvec)
        fix_colmax_kernel<true><<<g1, kFixThreads, sm, st>>>(A->n, w, X, ldx, part, large);
    else
        fix_colmax_kernel<false><<<g1, kFixThreads, sm, st>>>(A->n, w, X, ldx, part, large);
    if (!known) rc = check_launch();
    if (rc != CACG_OK) return rc;
    const int rpc = kFixThreads / a.cpr;
    const int g2 = (int)std::max<int64_t>(
        1, std::min<int64_t>((int64_t)sm_count() * 6, (A->n + 4 * rpc - 1) / (4 * rpc)));
    if (xvec)
        fix_convert_kernel<true><<<g2, kFixThreads, sm, st>>>(A->n, w, a.wp, X, ldx, part, g1, range,
                                                              (long long *)xi, scale, large);
    else
        fix_convert_kernel<false><<<g2, kFixThreads, sm, st>>>(A->n, w, a.wp, X, ldx, part, g1, range,
                                                               (long long *)xi, scale, large);
    rc = check_launch();
    if (rc != CACG_OK) return rc;
    const int64_t nblk = (A->n + (int64_t)a.runs * kFixR - 1) / ((int64_t)a.runs * kFixR);
    const unsigned blocks = (unsigned)std::min<int64_t>(nblk, std::min<int64_t>((int64_t)sm_count() * 3, kFixMaxBlocks));
    if (chain) {
        const int set = known ? chain->set ^ 1 : 1;
        a.ymax = parts + (size_t)set * kFixMaxBlocks * w;
        a.large0 = larges + (size_t)set * w;
        *chain = FixChain{Y, w, set, (int)blocks};
    }
    const int mode = !Z2 && (!Z1 || a.fold) ? (pow2 ? kFixPow2 : kFixNone)
                     : Z2 && cc == -1.0 && (!Z1 || a.fold) ? kFixStep
                                                           : kFixAny;
#define FIX_CASE(M)                                                              \
    case M:                                                                      \
        if (vec)                                                                 \
            fix_spmm_kernel<true, M><<<blocks, kFixThreads, sm, st>>>(a, A->dia);  \
        else                                                                     \
            fix_spmm_kernel<false, M><<<blocks, kFixThreads, sm, st>>>(a, A->dia); \
        break;
    switch (mode) {
        FIX_CASE(kFixPow2)
        FIX_CASE(kFixNone)
        FIX_CASE(kFixStep)
        FIX_CASE(kFixAny)
    }
#undef FIX_CASE
    return check_launch();
}

}  // namespace cacg
