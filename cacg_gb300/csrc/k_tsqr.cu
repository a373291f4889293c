// k_tsqr.cu -- tall-skinny QR of an n x k block (FP64): V = Q R with Q's
// columns orthonormal and R upper triangular with a positive diagonal.
//
// The reference names a TSQR (src/TSQR.c, src/TSQR.h) but its file is empty
// and its Householder QR (src/MatrixDecomposition.c:3-93) is unfinished and
// never called, so there is no reference behaviour to match; this is the
// GB300 form of the operation the s-step basis would use to orthonormalise a
// block.  It is CholeskyQR2 (Fukaya, Nakatsukasa, Yanagisawa, Yamamoto 2014):
//   G = V^T V,  R1 = chol(G) (upper),  Q1 = V R1^{-1},
//   G2 = Q1^T Q1, R2 = chol(G2),       Q  = Q1 R2^{-1},   R = R2 R1,
// which is orthogonal to working accuracy while the 2-norm condition number
// of V, its columns scaled to one norm, stays below about u^{-1/2} (1e8; the
// columns' own magnitudes do not count).  The Gram products are the library's
// (FP64 FMAs for few columns or rows, else digit planes on the tensor cores), the
// tall x small ones go by digit planes at every size, and the small Cholesky
// factors and triangular inverses run in one CTA.  A Cholesky pivot that is not
// positive and finite (V numerically rank-deficient) returns CACG_ERR_BREAKDOWN.
#include "cacg_internal.cuh"

namespace cacg {

constexpr int kQrMaxK = 128;
constexpr int kCholThreads = 512;

// One CTA: R = chol(G) (upper, G = R^T R) and Rinv = R^{-1}, both k x k
// row-major with zeros below the diagonal.  *bad gets kStatusBreakdown on a pivot that
// is not positive and finite (beside a kStatusTimeout of the product before).
//
// G = L D L^T by right-looking elimination with the same row operations applied
// to the identity, whose rows (L^{-1}) take the space below the diagonal: R =
// D^{1/2} L^T, R^{-1} = (L^{-1})^T D^{-1/2}.  On this part an FP64 division takes
// 340 clocks and each FP64 instruction its quadrant's pipe for 64, so a step has
// one division (in a warp a quadrant, for the multipliers), no square root (all of
// them at the end) and one FMA an element.  The form before, a square root and a
// division a step and then one thread a column of the inverse with a dependent FMA
// an element, took 155 us at k = 48 and 683 at 96; this 66 and
// 260 (the FP64 pipe of one SM, half of it lanes outside the triangles).
__global__ void __launch_bounds__(kCholThreads)
    chol_inv_kernel(int k, const double *__restrict__ G, double *__restrict__ R,
                    double *__restrict__ Rinv, int *__restrict__ bad) {
    extern __shared__ __align__(16) double qr_sm[];
    double *A = qr_sm;  // k x k
    __shared__ double t[kQrMaxK], sq[kQrMaxK], rs[kQrMaxK];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, kk = k * k;
    for (int i = tid; i < kk; i += kCholThreads) A[i] = G[i];
    __syncthreads();
    for (int j = 0; j < k; ++j) {
        const double *aj = A + (size_t)j * k;
        if (tid < kQrMaxK && (warp << 5) < k - j) {
            const double piv = aj[j];
            // positive and finite, on the bits (an FP64 comparison is 64 clocks of the chain)
            const uint32_t hi = (uint32_t)__double2hiint(piv);
            const bool ok = hi < 0x7ff00000u && (hi | (uint32_t)__double2loint(piv)) != 0u;
            const int l = j + tid;  // l = j: the pivot itself
            if (l > j && l < k) t[l] = ok ? aj[l] / piv : 0.0;
            if (tid == 0) {
                sq[j] = ok ? piv : 0.0;
                if (!ok) atomicOr(bad, kStatusBreakdown);
            }
        }
        __syncthreads();
        for (int i = j + 1 + warp; i < k; i += kCholThreads / 32) {
            const double ti = t[i];
            double *ai = A + (size_t)i * k;
            for (int c = lane; c < k; c += 32) {
                if (c < j || c >= i)
                    ai[c] = fma(-ti, aj[c], ai[c]);
                else if (c == j)
                    ai[c] = -ti;
            }
        }
        __syncthreads();
    }
    for (int i = tid; i < k; i += kCholThreads) {
        const double d = sqrt(sq[i]);
        sq[i] = d;
        rs[i] = 1.0 / d;
    }
    __syncthreads();
    for (int e = tid; e < kk; e += kCholThreads) {
        const int i = e / k, l = e % k;
        R[e] = l > i ? A[e] * rs[i] : l == i ? sq[i] : 0.0;
        Rinv[e] = l > i ? A[(size_t)l * k + i] * rs[l] : l == i ? rs[i] : 0.0;
    }
}

// R = A B for upper triangular k x k A, B: a CTA a row, an output a thread (one
// CTA for all rows: 26 us at k = 48, 294 at 128)
__global__ void triu_mul_kernel(int k, const double *__restrict__ A, const double *__restrict__ B,
                                double *__restrict__ R) {
    const int i = blockIdx.x;
    for (int c = threadIdx.x; c < k; c += blockDim.x) {
        double s = 0.0;
        for (int j = i; j <= c; ++j) s = fma(A[i * k + j], B[j * k + c], s);
        R[i * k + c] = c >= i ? s : 0.0;
    }
}

// the opt-in (set once per device) covers the largest k
constexpr int kQrSmemMax = kQrMaxK * kQrMaxK * (int)sizeof(double);

static int chol_inv(cudaStream_t st, int k, const double *G, double *R, double *Rinv, int *bad) {
    const int smem = (int)((size_t)k * k * sizeof(double));
    set_smem_attr(chol_inv_kernel, kQrSmemMax);
    chol_inv_kernel<<<1, kCholThreads, smem, st>>>(k, G, R, Rinv, bad);
    return check_launch();
}

}  // namespace cacg

using namespace cacg;

extern "C" int cacg_k_tsqr(int64_t n, int32_t k, const double *V, int64_t ldv, double *Q,
                           int64_t ldq, double *R, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < k || k <= 0 || k > kQrMaxK || !V || !Q || !R || ldv < k || ldq < k)
        return CACG_ERR_ARG;
    const size_t gws = (gram_workspace_bytes(n, k, k) + 255) / 256 * 256;
    const size_t q1b = ((size_t)n * k * sizeof(double) + 255) / 256 * 256;
    const size_t small = (size_t)5 * k * k * sizeof(double) + (size_t)k * sizeof(int);
    char *buf = nullptr;
    if (cudaMallocAsync((void **)&buf, gws + q1b + small + 256, st) != cudaSuccess) {
        cudaGetLastError();
        return CACG_ERR_OOM;
    }
    double *ws = (double *)buf;
    double *Q1 = (double *)(buf + gws);  // n x k, the first pass's factor
    double *G = (double *)(buf + gws + q1b), *R1 = G + (size_t)k * k, *R1i = R1 + (size_t)k * k,
           *R2 = R1i + (size_t)k * k, *R2i = R2 + (size_t)k * k;
    int *bad = (int *)(R2i + (size_t)k * k), *exps = bad + 1;
    int rc = cudaMemsetAsync(bad, 0, sizeof(int), st) == cudaSuccess ? CACG_OK : CACG_ERR_CUDA;
    // G = P^T P, and the exponents of P's columns for the product that follows
    auto gram = [&](const double *P, int64_t ldp) {
        ColExps ce;
        ce.L = exps;
        int r = launch_gram<double>(st, CACG_GRAM_AUTO, n, P, ldp, k, P, ldp, k, nullptr, 0, 0, G, k,
                                    nullptr, 0, ws, gws, true, &ce);
        if (r == CACG_OK && !ce.set)
            r = launch_col_exps(st, n, k, P, nullptr, ldp, ws, gws, exps, nullptr);
        return r;
    };
    // pass 1: G = V^T V, R1, Q1 = V R1^{-1}
    if (rc == CACG_OK) rc = gram(V, ldv);
    if (rc == CACG_OK) rc = chol_inv(st, k, G, R1, R1i, bad);
    if (rc == CACG_OK) rc = launch_tallsmall_x64(st, n, k, k, V, ldv, exps, R1i, k, Q1, k, bad);
    // pass 2: G2 = Q1^T Q1, R2, Q = Q1 R2^{-1}
    if (rc == CACG_OK) rc = gram(Q1, k);
    if (rc == CACG_OK) rc = chol_inv(st, k, G, R2, R2i, bad);
    if (rc == CACG_OK) rc = launch_tallsmall_x64(st, n, k, k, Q1, k, exps, R2i, k, Q, ldq, bad);
    if (rc == CACG_OK) {
        triu_mul_kernel<<<k, kQrMaxK, 0, st>>>(k, R2, R1, R);
        rc = check_launch();
    }
    int hb = 0;
    if (rc == CACG_OK) {
        if (cudaMemcpyAsync(&hb, bad, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            rc = CACG_ERR_CUDA;
    }
    cudaFreeAsync(buf, st);
    if (rc != CACG_OK) cudaGetLastError();  // a refused launch leaves no error behind
    if (rc == CACG_OK && hb) rc = hb & kStatusTimeout ? CACG_ERR_TIMEOUT : CACG_ERR_BREAKDOWN;
    return rc;
}
