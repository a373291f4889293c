// k_lu.cu -- the small dense solve of the CA iteration, in FP64.
//
// Reference operation replaced (sclc/cacg): LUsolver_v1_KeeplhsMat,
// src/DLSsolvers.c:106-208 -- Crout LU with unit-diagonal U and NO pivoting
// (reciprocal of the pivot times the pivot row, then the trailing update),
// forward substitution dividing by L's diagonal through a reciprocal, back
// substitution with U's unit diagonal.  The same elimination order is kept
// so the GPU result matches the reference to rounding.
//
// The reference refactors Q^T AQ inside every call (twice per iteration:
// for alpha, and one iteration later for beta); here the factor of each
// Q^T AQ is computed once and reused by both solves.
//
// The factor F is 2*k*k + k doubles: the Crout factors, the reciprocals of
// L's diagonal (the reference multiplies by 1/L_ii, src/DLSsolvers.c:168),
// and the factors again, transposed, for the column-sweep solves.
// A zero or non-finite pivot sets *status = 1 (CACG_ERR_BREAKDOWN at the
// host) instead of trapping; the arithmetic continues as the reference's
// does (inf/NaN propagate) and the host stops the iteration.
#include <cooperative_groups.h>

#include "cacg_internal.cuh"
#include "lu_block.cuh"

namespace cacg {

namespace cgrp = cooperative_groups;

constexpr int kLuThreads = 512;
constexpr int kLuSmemK = 144;  // factor in shared memory up to k = 144 (162 KB)

// One CTA.  W is the working matrix: shared memory when it fits, else F.
__global__ void __launch_bounds__(kLuThreads)
    lu_factor_kernel(int k, const double *__restrict__ M, double *__restrict__ F,
                     int *__restrict__ status, int use_smem) {
    extern __shared__ __align__(16) double Ws[];
    double *W = use_smem ? Ws : F;
    const int kk = k * k;
    for (int i = threadIdx.x; i < kk; i += blockDim.x) W[i] = M[i];
    __syncthreads();
    int bad = 0;
    double *Dinv = F + (size_t)kk;  // reciprocals of L's diagonal, read by the solves
    for (int d = 0; d < k; ++d) {
        // warp 0 scales the pivot row; one FP64 division per step
        if (threadIdx.x < 32) {
            double inv = 0.0;
            if (threadIdx.x == 0) {
                const double piv = W[d * k + d];
                if (piv == 0.0 || !isfinite(piv)) bad = 1;
                inv = 1.0 / piv;
                Dinv[d] = inv;
            }
            inv = __shfl_sync(0xffffffffu, inv, 0);
            for (int c = d + 1 + threadIdx.x; c < k; c += 32) W[d * k + c] *= inv;
        }
        __syncthreads();
        // trailing update, rows by warp, columns by lane (no index division)
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        for (int i = d + 1 + warp; i < k; i += kLuThreads / 32) {
            const double lid = W[i * k + d];
            for (int c = d + 1 + lane; c < k; c += 32)
                W[i * k + c] = W[i * k + c] - lid * W[d * k + c];
        }
        __syncthreads();
    }
    if (use_smem)
        for (int i = threadIdx.x; i < kk; i += blockDim.x) F[i] = W[i];
    // transposed copy for the column-sweep solves: FT[i][j] = F[j][i]
    double *FT = F + (size_t)kk + k;
    for (int idx = threadIdx.x; idx < kk; idx += blockDim.x) {
        const int i = idx / k, j = idx % k;
        FT[idx] = W[(size_t)j * k + i];
    }
    if (threadIdx.x == 0 && bad && status) atomicOr(status, kStatusBreakdown);
}

// The same factor spread over a cluster of kLucCtas CTAs (one SM each): CTA r
// owns rows i = r (mod kLucCtas) in its shared memory.  Step d: the owner of
// row d scales it by the pivot's reciprocal; one cluster barrier; every CTA
// copies the scaled row d from the owner's shared memory (distributed shared
// memory) and updates its rows i > d.  Every element sees the same
// operations in the same order as lu_factor_kernel (bit-identical factors);
// the trailing update's FP64 work is split over kLucCtas SMs' FP64 pipes.
constexpr int kLucCtas = 8;
constexpr int kLucThreads = 256;
constexpr int kLucMaxK = 256;

__global__ void __cluster_dims__(kLucCtas, 1, 1) __launch_bounds__(kLucThreads)
    lu_factor_cluster_kernel(int k, const double *__restrict__ M, double *__restrict__ F,
                             int *__restrict__ status) {
    extern __shared__ __align__(16) double luc_sm[];
    cgrp::cluster_group cluster = cgrp::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int nloc = (k - rank + kLucCtas - 1) / kLucCtas;  // rows rank, rank + C, ...
    const int rows_max = (k + kLucCtas - 1) / kLucCtas;
    double *Wl = luc_sm;                        // nloc x k: local rows
    double *prow = luc_sm + (size_t)rows_max * k;  // the current pivot row
    for (int idx = threadIdx.x; idx < nloc * k; idx += blockDim.x) {
        const int li = idx / k, c = idx - li * k;
        Wl[idx] = M[(size_t)(li * kLucCtas + rank) * k + c];
    }
    double *Dinv = F + (size_t)k * k;
    int bad = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    for (int d = 0; d < k; ++d) {
        const int owner = d % kLucCtas;
        if (rank == owner && warp == 0) {
            double *rd = Wl + (size_t)(d / kLucCtas) * k;
            double inv = 0.0;
            if (lane == 0) {
                const double piv = rd[d];
                if (piv == 0.0 || !isfinite(piv)) bad = 1;
                inv = 1.0 / piv;
                Dinv[d] = inv;
            }
            inv = __shfl_sync(0xffffffffu, inv, 0);
            for (int c = d + 1 + lane; c < k; c += 32) rd[c] *= inv;
        }
        cluster.sync();  // row d scaled, visible to the cluster
        const double *src = cluster.map_shared_rank(Wl + (size_t)(d / kLucCtas) * k, owner);
        for (int c = d + 1 + threadIdx.x; c < k; c += blockDim.x) prow[c] = src[c];
        __syncthreads();
        // local rows i > d: rows by warp, columns by lane
        const int li0 = (d + 1 - rank + kLucCtas - 1) / kLucCtas;  // first local row past d
        for (int li = li0 + warp; li < nloc; li += kLucThreads / 32) {
            double *wi = Wl + (size_t)li * k;
            const double lid = wi[d];
            for (int c = d + 1 + lane; c < k; c += 32) wi[c] = wi[c] - lid * prow[c];
        }
        __syncthreads();
    }
    // factors and their transpose (the column-sweep solves read FT)
    double *FT = F + (size_t)k * k + k;
    for (int idx = threadIdx.x; idx < nloc * k; idx += blockDim.x) {
        const int li = idx / k, c = idx - li * k;
        const int i = li * kLucCtas + rank;
        F[(size_t)i * k + c] = Wl[idx];
        FT[(size_t)c * k + i] = Wl[idx];
    }
    if (threadIdx.x == 0 && bad && status) atomicOr(status, kStatusBreakdown);
    cluster.sync();  // no CTA leaves while another may still read its rows
}

// The cluster factor with the pivot rows pushed instead of pulled: CTA r owns
// rows i = r (mod kLucCtas); the owner of row d + 1 updates it at step d ahead of
// its other rows, takes the pivot and scales the row into U's, and writes it with
// st.async into every CTA's copy of U, whose mbarrier of that row the bytes
// complete.  No cluster barrier per step: the chain is one FMA, the division (340
// clocks; an FMA is 64 on this part whatever the lanes), one product and the
// transfer; the trailing update runs beside it.  Warp 0 holds the pivot alone on
// its quadrant's FP64 pipe (warp 4 rests while this CTA takes a pivot).  Every
// element sees the operations of lu_factor_kernel in the same order
// (bit-identical factors).  k = 96: 69.5 us, k = 128: 117 (pulled: 135, 195).
constexpr int kLupThreads = 256;
constexpr int kLupMinK = 48;
constexpr int kLupMaxK = 160;  // U (k x k) and the local rows in shared memory
constexpr long long kLupPolls = 1ll << 22;

__device__ __forceinline__ unsigned lup_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned lup_map(unsigned a, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ bool lup_wait(uint64_t *bar) {
    for (long long i = 0; i < kLupPolls; ++i) {
        unsigned ok;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(lup_u32(bar))
            : "memory");
        if (ok) return true;
    }
    return false;
}

__global__ void __cluster_dims__(kLucCtas, 1, 1) __launch_bounds__(kLupThreads)
    lu_factor_push_kernel(int k, const double *__restrict__ M, double *__restrict__ F,
                          int *__restrict__ status) {
    extern __shared__ __align__(16) double lup_sm[];
    __shared__ double s_inv;
    __shared__ int s_bad;
    cgrp::cluster_group cluster = cgrp::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int nloc = (k - rank + kLucCtas - 1) / kLucCtas;
    const int rows_max = (k + kLucCtas - 1) / kLucCtas;
    double *U = lup_sm;                       // k x k: scaled pivot rows, columns past the pivot
    double *Wl = U + (size_t)k * k;           // nloc x k: local rows
    uint64_t *bar = reinterpret_cast<uint64_t *>(Wl + (size_t)rows_max * k);  // row d has arrived
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double *Dinv = F + (size_t)k * k;
    for (int idx = tid; idx < nloc * k; idx += kLupThreads) {
        const int li = idx / k, c = idx - li * k;
        Wl[idx] = M[(size_t)(li * kLucCtas + rank) * k + c];
    }
    for (int d = tid; d < k; d += kLupThreads) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(lup_u32(&bar[d])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile(
            "{\n"
            ".reg .b64 st;\n"
            "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n"
            "}\n" ::"r"(lup_u32(&bar[d])),
            "r"(8 * (k - 1 - d))
            : "memory");
    }
    if (tid == 0) s_bad = 0;
    __syncthreads();
    cluster.sync();  // every CTA's barriers expect their bytes

    // warps 0 .. 3: row r updated with row d (d < 0: as it is), its pivot taken,
    // scaled and pushed
    auto pivot_row = [&](int r, int d) {
        double *wr = Wl + (size_t)(r / kLucCtas) * k;
        const double l = d >= 0 ? wr[d] : 0.0;
        const double *ud = U + (size_t)(d >= 0 ? d : 0) * k;
        double w[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = r + tid + 128 * e;
            w[e] = c < k ? wr[c] : 0.0;
            if (c < k && d >= 0) w[e] = fma(-l, ud[c], w[e]);
        }
        if (warp == 0) {
            const double piv = __shfl_sync(0xffffffffu, w[0], 0);
            const double inv = 1.0 / piv;
            if (lane == 0) {
                s_inv = inv;
                Dinv[r] = inv;
                if (lu_bad_pivot(piv)) s_bad = 1;
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const double inv = s_inv;
        const unsigned mb = lup_u32(&bar[r]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = r + tid + 128 * e;
            if (c >= k) break;
            if (c == r) {
                wr[c] = w[e];
                continue;
            }
            const double u = w[e] * inv;
            wr[c] = u;
            const unsigned dst = lup_u32(U + (size_t)r * k + c);
#pragma unroll
            for (unsigned q = 0; q < (unsigned)kLucCtas; ++q)
                asm volatile(
                    "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, "
                    "[%2];" ::"r"(lup_map(dst, q)),
                    "l"(__double_as_longlong(u)), "r"(lup_map(mb, q))
                    : "memory");
        }
    };

    bool ok = true;
    if (rank == 0 && warp < 4) pivot_row(0, -1);
    for (int d = 0; d + 1 < k; ++d) {
        ok = lup_wait(&bar[d]);
        if (__syncthreads_or(!ok)) {  // (also: the last step's rows are written)
            ok = false;
            break;
        }
        const bool mine = (d + 1) % kLucCtas == rank;
        const double *ud = U + (size_t)d * k;
        const int li0 = (d + 1 - rank + kLucCtas - 1) / kLucCtas + (mine ? 1 : 0);
        if (mine && warp < 4) {
            pivot_row(d + 1, d);
        } else if (!mine || warp != 4) {
            // local rows past the next pivot row: rows by warp, columns by lane
            const int nw = mine ? 3 : kLupThreads / 32, w0 = mine ? warp - 5 : warp;
            for (int li = li0 + w0; li < nloc; li += nw) {
                double *wi = Wl + (size_t)li * k;
                const double l = wi[d];
                for (int c = d + 1 + lane; c < k; c += 32) wi[c] = fma(-l, ud[c], wi[c]);
            }
        }
    }
    __syncthreads();
    double *FT = F + (size_t)k * k + k;
    for (int idx = tid; idx < nloc * k; idx += kLupThreads) {
        const int li = idx / k, c = idx - li * k;
        const int i = li * kLucCtas + rank;
        F[(size_t)i * k + c] = Wl[idx];
        FT[(size_t)c * k + i] = Wl[idx];
    }
    if (tid == 0 && status) {
        if (s_bad) atomicOr(status, kStatusBreakdown);
        if (!ok) atomicOr(status, kStatusTimeout);
    }
    cluster.sync();  // no CTA leaves while another may still write into it
}

// One CTA (lu_block.cuh) for the small factors, where eight SMs' transfers cost
// more than their FP64 pipes give.
constexpr int kLuLaMaxK = 128;  // k x k doubles in shared memory (128 KB)

__global__ void __launch_bounds__(kLuBlockThreads)
    lu_factor_la_kernel(int k, const double *__restrict__ M, double *__restrict__ F,
                        int *__restrict__ status) {
    extern __shared__ __align__(16) double lw[];
    __shared__ double s_inv;
    __shared__ int s_bad;
    const int kk = k * k, tid = threadIdx.x;
    if (tid == 0) s_bad = 0;
    for (int i = tid; i < kk; i += blockDim.x) lw[i] = M[i];
    __syncthreads();
    lu_factor_block(lw, k, F + (size_t)kk, &s_inv, &s_bad);
    double *FT = F + (size_t)kk + k;
    for (int idx = tid; idx < kk; idx += blockDim.x) {
        const int i = idx / k, j = idx - i * k;
        F[idx] = lw[idx];
        FT[idx] = lw[(size_t)j * k + i];
    }
    if (tid == 0 && s_bad && status) atomicOr(status, kStatusBreakdown);
}

// Y (k x r) from the factor F (k*k factors + k reciprocal diagonal) and RHS
// (k x r).  Each CTA solves kLuRC columns with kLuTPC threads per column
// splitting the inner products; many CTAs spread the FP64 work over SMs.
constexpr int kLuRC = 8;    // right-hand-side columns per CTA
constexpr int kLuTPC = 16;  // threads per column

__global__ void __launch_bounds__(kLuRC * kLuTPC)
    lu_solve_kernel(int k, const double *__restrict__ F, int r, const double *__restrict__ RHS,
                    double *__restrict__ Y, int use_smem) {
    extern __shared__ __align__(16) double sm[];
    double *Fs = use_smem ? sm : nullptr;
    double *Z = sm + (use_smem ? (size_t)k * k + k : 0);  // k x kLuRC
    const double *Fm = use_smem ? Fs : F;
    if (use_smem)
        for (int i = threadIdx.x; i < k * k + k; i += blockDim.x) Fs[i] = F[i];
    const int c0 = blockIdx.x * kLuRC;
    const int cl = threadIdx.x / kLuTPC, sub = threadIdx.x % kLuTPC;
    const int col = c0 + cl;
    const bool active = col < r;
    for (int i = threadIdx.x; i < k * kLuRC; i += blockDim.x) {
        int row = i / kLuRC, cc = i % kLuRC;
        Z[i] = (c0 + cc < r) ? RHS[(size_t)row * r + c0 + cc] : 0.0;
    }
    __syncthreads();
    // forward: Z[i] = (Z[i] - sum_{q<i} L[i][q] Z[q]) * (1 / L[i][i])
    for (int i = 0; i < k; ++i) {
        double s = 0.0;
        for (int q = sub; q < i; q += kLuTPC) s = fma(Fm[i * k + q], Z[q * kLuRC + cl], s);
#pragma unroll
        for (int o = kLuTPC / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, kLuTPC);
        if (sub == 0 && active) Z[i * kLuRC + cl] = (Z[i * kLuRC + cl] - s) * Fm[k * k + i];
        __syncthreads();
    }
    // backward: Y[i] = Z[i] - sum_{q>i} U[i][q] Y[q]   (U unit diagonal)
    for (int i = k - 2; i >= 0; --i) {
        double s = 0.0;
        for (int q = i + 1 + sub; q < k; q += kLuTPC) s = fma(Fm[i * k + q], Z[q * kLuRC + cl], s);
#pragma unroll
        for (int o = kLuTPC / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, kLuTPC);
        if (sub == 0 && active) Z[i * kLuRC + cl] = Z[i * kLuRC + cl] - s;
        __syncthreads();
    }
    for (int i = threadIdx.x; i < k * kLuRC; i += blockDim.x) {
        int row = i / kLuRC, cc = i % kLuRC;
        if (c0 + cc < r) Y[(size_t)row * r + c0 + cc] = Z[i];
    }
}

// Column-sweep ("axpy") triangular solves, ceil(k / 32) warps per right-hand
// side (lu_block.cuh), a warp per quadrant of the SM.  Same arithmetic as the
// substitution above, summed column by column (agrees with the reference to
// rounding).
__global__ void __launch_bounds__(160)
    lu_solve_sweep_kernel(int k, int nt, int cols, const double *__restrict__ F, int r,
                          const double *__restrict__ RHS, double *__restrict__ Y) {
    __shared__ double ys[4][160];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = warp / nt, w = warp % nt;
    const int c = blockIdx.x * cols + g;
    if (c >= r) return;  // whole groups of warps; no block-wide barrier follows
    const int j = 32 * w + lane;
    const double z = j < k ? RHS[(size_t)j * r + c] : 0.0;
    const double y = lu_sweep(k, nt, w, lane, 1 + g, z, F + (size_t)k * k, F + (size_t)k * k + k,
                              ys[g]);
    if (j < k) Y[(size_t)j * r + c] = y;
}

int launch_lu_factor(cudaStream_t st, int k, const double *M, double *F, int *status) {
    if (k <= 0) return CACG_ERR_ARG;
    // factor and one solve, one CTA / pulled rows before, pushed rows now: k = 44
    // 46.8 and 51.5 us; k = 64 77 and 68; k = 96 169 and 107; k = 128 248 and 172;
    // k = 160 321 and 241.  Above, U does not fit beside the local rows.
    if (k >= kLupMinK && k <= kLupMaxK) {
        const size_t psmem = ((size_t)k * k + (size_t)((k + kLucCtas - 1) / kLucCtas) * k + k) *
                             sizeof(double);
        const size_t room = max_smem_optin() - 64;  // beside the kernel's static variables
        set_smem_attr(lu_factor_push_kernel, (int)room);
        if (psmem <= room) {
            lu_factor_push_kernel<<<kLucCtas, kLupThreads, psmem, st>>>(k, M, F, status);
            if (cudaPeekAtLastError() == cudaSuccess) return check_launch();
            cudaGetLastError();  // cluster launch refused: the pulling factors below
        }
    }
    if (k <= 64) {
        const size_t smem = (size_t)k * k * sizeof(double);
        set_smem_attr(lu_factor_la_kernel, kLuLaMaxK * kLuLaMaxK * (int)sizeof(double));
        lu_factor_la_kernel<<<1, kLuBlockThreads, smem, st>>>(k, M, F, status);
        return check_launch();
    }
    if (k >= kLucCtas && k <= kLucMaxK) {
        const size_t csmem = ((size_t)((k + kLucCtas - 1) / kLucCtas) * k + k) * sizeof(double);
        set_smem_attr(lu_factor_cluster_kernel, (int)(((size_t)(kLucMaxK / kLucCtas) * kLucMaxK + kLucMaxK) * sizeof(double)));
        lu_factor_cluster_kernel<<<kLucCtas, kLucThreads, csmem, st>>>(k, M, F, status);
        if (cudaPeekAtLastError() == cudaSuccess) return check_launch();  // counted
        cudaGetLastError();  // cluster launch refused: the one-CTA factor below
    }
    int use_smem = k <= kLuSmemK;
    size_t smem = use_smem ? (size_t)k * k * sizeof(double) : 0;
    set_smem_attr(lu_factor_kernel, (int)max_smem_optin());
    lu_factor_kernel<<<1, kLuThreads, smem, st>>>(k, M, F, status, use_smem);
    return check_launch();
}

int launch_lu_solve(cudaStream_t st, int k, const double *F, int r, const double *RHS,
                    double *Y) {
    if (k <= 0 || r <= 0) return CACG_ERR_ARG;
    if (k <= 160) {
        const int nt = (k + 31) / 32, cols = nt >= 3 ? 1 : 4 / nt;
        lu_solve_sweep_kernel<<<(r + cols - 1) / cols, 32 * nt * cols, 0, st>>>(k, nt, cols, F, r,
                                                                                RHS, Y);
        return check_launch();
    }
    size_t zbytes = (size_t)k * kLuRC * sizeof(double);
    size_t fbytes = ((size_t)k * k + k) * sizeof(double);
    int use_smem = (fbytes + zbytes) <= max_smem_optin() - 1024;
    size_t smem = zbytes + (use_smem ? fbytes : 0);
    if (smem > max_smem_optin()) return CACG_ERR_UNSUPPORTED;
    set_smem_attr(lu_solve_kernel, (int)max_smem_optin());
    int blocks = (r + kLuRC - 1) / kLuRC;
    lu_solve_kernel<<<blocks, kLuRC * kLuTPC, smem, st>>>(k, F, r, RHS, Y, use_smem);
    return check_launch();
}

}  // namespace cacg

using namespace cacg;

extern "C" int cacg_k_lu(int32_t k, const double *M, int32_t r, const double *RHS, double *Y,
                         int *status, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    double *F = nullptr;
    if (cudaMallocAsync((void **)&F, ((size_t)2 * k * k + k) * sizeof(double), st) != cudaSuccess)
        return CACG_ERR_OOM;
    int rc = launch_lu_factor(st, k, M, F, status);
    if (rc == CACG_OK) rc = launch_lu_solve(st, k, F, r, RHS, Y);
    cudaFreeAsync(F, st);
    return rc;
}
