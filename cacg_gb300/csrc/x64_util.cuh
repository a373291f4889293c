// x64_util.cuh -- FP64 values as fp16 digit planes, for FP64 products on the
// fp16 tensor cores (k_gram_x64.cu, k_tsm_x64.cu).
//
// The products follow the splitting of Ozaki, Ogita, Oishi and Rump
// ("Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", Numer. Algorithms 59, 2012) with
// integer digits: a vector that shares one scale (a column over a row chunk,
// or a row) becomes X = round(x 2^(1077 - E)), |X| <= 2^55, E the biased
// exponent of its largest element, and X = sum_i d_i 2^(8 i), i = 0 .. 6,
// with balanced digits d_i in [-128, 128].  A digit is exact in fp16, a
// product of two digits is at most 2^14, and a sum of up to 2^10 of them is an
// integer below 2^24, exact in the FP32 accumulator.  Plane p holds digit
// 6 - p; the 28 plane products with p + q <= 6 are kept (the dropped ones are
// below 2^-56 of the largest product), accumulated per p + q.  So each sum is
// exact up to the rounding of X at 2^-55 of its vector's largest element and
// the dropped products.  That error goes with the largest elements of the two
// vectors, an FMA chain's with the elements that are multiplied: for vectors of even
// magnitude it is the smaller one, for graded ones it need not be.  Each kernel
// says what keeps it there: k_gram_x64.cu a line beyond which a chunk takes FMAs,
// k_tsm_x64.cu an exponent per column of the tall operand.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace cacg {

constexpr int kXPlanes = 7;
constexpr int kXMinExp = 64;  // smallest biased exponent of a scale (below: FP64 path)

// |x|'s high word as an ordered key of its magnitude (a nonzero value below
// 2^-1042 counts as 1, so a key of 0 means +-0)
__device__ __forceinline__ uint32_t x64_key(double x) {
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    const uint32_t l = (uint32_t)__double2loint(x);
    return h | (l != 0u ? 1u : 0u);
}

// scale exponent of a vector whose largest key is `key`; *bad when the digits
// cannot hold it (Inf, NaN, or a largest magnitude below 2^-959)
__device__ __forceinline__ int x64_scale(uint32_t key, bool *bad) {
    const int e = (int)(key >> 20);
    if (e >= 0x7ff || (e < kXMinExp && key != 0u)) *bad = true;
    return e < kXMinExp ? kXMinExp : e;
}

// A column's exponent for the tall x small products: of about its 2-norm, from the
// maxima of its row groups (emax: ngroups x kc keys, column c), at least that of its
// largest element; 1023 for a zero column and one with Inf or NaN.  Called by 16
// threads a column (q) of a block, sh their shared scratch.
__device__ __forceinline__ void x64_col_exp(const uint32_t *__restrict__ emax, int ngroups, int kc,
                                            int c, bool on, int el, int q, float (*sh)[32],
                                            int *__restrict__ out) {
    uint32_t *shk = reinterpret_cast<uint32_t *>(&sh[0][0]);
    uint32_t k = 0u;
    if (on)
        for (int g = q; g < ngroups; g += 16) k = max(k, emax[(size_t)g * kc + c]);
    shk[q * 32 + el] = k;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) k = max(k, shk[i * 32 + el]);
    __syncthreads();
    const int E = (int)(k >> 20);
    float s = 0.f;
    if (on && k != 0u && E < 0x7ff)
        for (int g = q; g < ngroups; g += 16) {
            const int d = 2 * (E - (int)(emax[(size_t)g * kc + c] >> 20));
            if (d < 127) s += __uint_as_float((uint32_t)(127 - d) << 23);  // 2^-d
        }
    sh[q][el] = s;
    __syncthreads();
    if (q == 0 && on) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) t += sh[i][el];
        // t >= 1: half its binary logarithm
        const int h = ((int)(__float_as_uint(t) >> 23) - 126) >> 1;
        *out = k == 0u || E >= 0x7ff ? 1023 : min(E + max(h, 0), 2046);
    }
}

// the seven balanced digits of x at scale E (E20: in units of 2^-20, E at least x's
// exponent, and 64 for a zero), biased by 128: bytes 0 .. 5 of (hi, lo) are d_0 + 128
// .. d_5 + 128, the top 16 bits d_6 + 128 (0 .. 256)
__device__ __forceinline__ void x64_digits(double x, uint32_t E20, uint32_t &lo, uint32_t &hi) {
    const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
    const uint32_t s = (E20 - (xh & 0x7ff00000u)) >> 20;
    const uint32_t mh = (xh & 0xfffffu) | 0x100000u;
    uint64_t m;  // 8 x the 53-bit significand, shifted right (by 64 or more: 0): 2 |X|, a bit to round on
    const uint64_t m8 = ((uint64_t)__funnelshift_l(xl, mh, 3) << 32) | (uint64_t)(xl << 3);
    asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m8), "r"(s));
    const uint32_t sg = (uint32_t)((int32_t)xh >> 31);
    const uint32_t a = (uint32_t)m ^ sg, b = (uint32_t)(m >> 32) ^ sg;
    // 2 sum_i 128 2^(8 i) + 1, the 1 rounding a positive half up and completing a
    // negative value's two's complement (whose floor rounds its half away); halved
    const uint64_t v = ((((uint64_t)b << 32) | a) + 0x0101010101010101ull) >> 1;
    lo = (uint32_t)v;
    hi = (uint32_t)(v >> 32);
}

// plane words of two values at scales E0, E1 (units of 2^-20): w[p] = {digit 6-p of x0 (low half), of x1 (high half)} as fp16
__device__ __forceinline__ void x64_planes2(double x0, double x1, uint32_t E0, uint32_t E1,
                                            uint32_t (&w)[kXPlanes]) {
    uint32_t l0, h0, l1, h1;
    x64_digits(x0, E0, l0, h0);
    x64_digits(x1, E1, l1, h1);
    // bytes (x0 digit i, x1 digit i, x0 digit i+1, x1 digit i+1)
    const uint32_t d01 = __byte_perm(l0, l1, 0x5140), d23 = __byte_perm(l0, l1, 0x7362);
    const uint32_t d45 = __byte_perm(h0, h1, 0x5140), d6 = __byte_perm(h0, h1, 0x7632);
    // 0x6400 | byte is 1024 + byte in fp16; minus 1152 leaves the digit, exactly
    const uint32_t k64 = 0x64646464u;
    uint32_t u[kXPlanes] = {d6 | 0x64006400u,               __byte_perm(d45, k64, 0x4342),
                            __byte_perm(d45, k64, 0x4140), __byte_perm(d23, k64, 0x4342),
                            __byte_perm(d23, k64, 0x4140), __byte_perm(d01, k64, 0x4342),
                            __byte_perm(d01, k64, 0x4140)};
#pragma unroll
    for (int p = 0; p < kXPlanes; ++p)
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(w[p]) : "r"(u[p]), "r"(0x64806480u));
}

// h 2^32 + l as FP64, rounded once (|h|, |l| < 2^50): both are put into a
// double's significand by integer additions, so the FP64 pipe does two additions
// (a conversion from 64 bits holds it for several times as long)
__device__ __forceinline__ double x64_join(long long h, long long l) {
    const double a = __longlong_as_double(0x4538000000000000ll + h);  // 1.5 2^84 + h 2^32
    const double b = __longlong_as_double(0x4338000000000000ll + l);  // 1.5 2^52 + l
    return (a - (0x1.8p84 + 0x1.8p52)) + b;                           // the difference is exact
}

// v as FP64, rounded to nearest (ties away from zero), by integer instructions
// alone: for kernels whose FP64 pipe is the busier one
__device__ __forceinline__ double x64_from_ll(long long v) {
    const unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    const int z = __clzll((long long)m);
    const unsigned long long u = m << (z & 63);  // leading bit at 63 (0 for 0)
    // the leading bit of u >> 11 adds one to the exponent field, and so does a rounding carry
    const unsigned long long r = (u >> 11) + ((u >> 10) & 1ull);
    const uint32_t e = u ? (uint32_t)(1023 + 62 - z) << 20 : 0u;
    return __hiloint2double((int)(((uint32_t)(r >> 32) + e) | ((uint32_t)(v >> 32) & 0x80000000u)),
                            (int)(uint32_t)r);
}

// t 2^sc, the power of two added to the exponent field (|sc| < 900, |t| between 1
// and 2^79, or `zero`)
__device__ __forceinline__ double x64_scaled(double t, bool zero, int sc) {
    return zero ? 0.0 : __hiloint2double(__double2hiint(t) + (sc << 20), __double2loint(t));
}

// Instruction descriptor of kind::f16 with fp16 inputs and FP32 accumulation
__host__ __device__ constexpr unsigned x64_idesc(int M, int N) {
    return (1u << 4) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}

}  // namespace cacg
