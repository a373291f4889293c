// lu_block.cuh -- the small no-pivot Crout factor on one CTA (k_lu.cu, k_batch.cu).
#pragma once

#include <stdint.h>

namespace cacg {

constexpr int kLuBlockThreads = 512;

// W (k x k, shared memory) <- its factors (U unit-diagonal, row i scaled by its
// pivot's reciprocal past the diagonal), Dinv[i] the reciprocals; *s_bad is set
// on a zero or non-finite pivot.  Every element sees the operations of the
// right-looking elimination in its order (src/DLSsolvers.c:106-208), whatever
// the thread layout.
//
// On this part an FP64 instruction holds its quadrant's pipe for 64 clocks and a
// division takes 340, so a step costs at least one FMA, the division and one
// product in sequence.  Warp 0 has that chain to itself on quadrant 0; warps 1-3
// hold the pivot row's columns past the first 32; the trailing rows are updated
// beside it by the other warps of quadrants 1-3, and by quadrant 0's too while the
// trailing matrix is what bounds the step (more than kLuWide columns).  One
// barrier a step.  k = 44: 30 us (33 with one warp for the pivot row and the
// trailing rows on all quadrants), the chain's 44 x 0.35 us and the hand-overs.
constexpr int kLuWide = 40;

// zero or non-finite, on the bits (an FP64 comparison is 64 clocks of the chain)
__device__ __forceinline__ bool lu_bad_pivot(double p) {
    const uint32_t h = (uint32_t)__double2hiint(p) & 0x7fffffffu;
    return h >= 0x7ff00000u || (h | (uint32_t)__double2loint(p)) == 0u;
}

__device__ __forceinline__ void lu_factor_block(double *W, int k, double *Dinv, double *s_inv,
                                                int *s_bad) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // warps 0-3: row r updated with row d (d < 0: as it is), its pivot, scaled
    auto pivot_row = [&](int r, int d) {
        double *wr = W + (size_t)r * k;
        const int c = r + tid;
        const bool on = c < k;
        double w = on ? wr[c] : 0.0;
        if (on && d >= 0) w = fma(-wr[d], W[(size_t)d * k + c], w);
        if (warp == 0) {
            const double piv = __shfl_sync(0xffffffffu, w, 0);
            const double inv = 1.0 / piv;
            if (lane == 0) {
                *s_inv = inv;
                Dinv[r] = inv;
                if (lu_bad_pivot(piv)) *s_bad = 1;
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (on) wr[c] = c == r ? w : w * *s_inv;
    };
    if (warp < 4) pivot_row(0, -1);
    __syncthreads();
    for (int d = 0; d + 1 < k; ++d) {
        const int x = k - d - 1;  // trailing columns d + 1 .. k - 1
        if (warp < 4) {
            pivot_row(d + 1, d);
        } else {
            // rows d + 2 ..: entry e = q x + r, q = floor(e / x) by the high word of
            // e * ceil(2^32 / x) (exact for e < 2^32 / x)
            const bool wide = x > kLuWide;
            const int wk = wide ? warp - 4 : ((warp & 3) == 0 ? -1 : (warp >> 2) * 3 + (warp & 3) - 4);
            const int nw = wide ? kLuBlockThreads / 32 - 4 : (kLuBlockThreads / 32 - 4) / 4 * 3;
            if (wk >= 0) {
                const double *U = W + (size_t)d * k;
                const uint32_t mg = x > 1 ? 0xFFFFFFFFu / (uint32_t)x + 1u : 0u;
                for (int e = 32 * wk + lane; e < (x - 1) * x; e += 32 * nw) {
                    const int q = x > 1 ? (int)__umulhi((uint32_t)e, mg) : e;
                    double *wr = W + (size_t)(d + 2 + q) * k;
                    const int c = d + 1 + (e - q * x);
                    wr[c] = fma(-wr[d], U[c], wr[c]);
                }
            }
        }
        __syncthreads();
    }
}

// Column-sweep solves of one right-hand side by nt = ceil(k / 32) warps, warp w
// of them holding rows 32 w .. 32 w + 31 in z (one a lane): forward, y_i = z_i /
// L_ii through the stored reciprocal, then z_j -= L_ji y_i for j > i; backward with
// U's unit diagonal, z_j -= U_ji x_i for j < i (src/DLSsolvers.c:156-207), every
// row in the order of i.  The warp that owns a block of 32 rows walks its chain
// (a product and an FMA a step forward, an FMA backward: 64 clocks each) and hands
// kLuSub values at a time to the others through ys, which apply them while it
// walks on; one warp holding all rows pays an FMA per 32 rows at every step
// (k = 128: 54 us, 28 here; k = 96: 33 and 21; k = 20: 8.0 and 6.5).  FT: the factors
// transposed (global or shared memory), read a hand-over ahead.
constexpr int kLuSub = 8;

__device__ __forceinline__ double lu_sweep(int k, int nt, int w, int lane, int barrier, double z,
                                           const double *__restrict__ Dinv,
                                           const double *__restrict__ FT, double *ys) {
    const int j = 32 * w + lane;
    const int nsub = (k + kLuSub - 1) / kLuSub;
    const double dinv = j < k ? Dinv[j] : 0.0;
    auto sync = [&]() {
        if (nt > 1)
            asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(32 * nt) : "memory");
        else
            __syncwarp();
    };
    double cn[kLuSub], c[kLuSub];
    auto load = [&](int sb) {
#pragma unroll
        for (int u = 0; u < kLuSub; ++u) {
            const int i = kLuSub * sb + u;
            cn[u] = i < k && j < k ? FT[(size_t)i * k + j] : 0.0;
        }
    };
    // forward: hand-over sb covers rows kLuSub sb ..; blocks before it are done
    load(0);
    for (int sb = 0; sb < nsub; ++sb) {
        const int i0 = kLuSub * sb, own = i0 >> 5;
#pragma unroll
        for (int u = 0; u < kLuSub; ++u) c[u] = cn[u];
        if (sb + 1 < nsub) load(sb + 1);
        if (w == own) {
#pragma unroll
            for (int u = 0; u < kLuSub; ++u) {
                if (i0 + u >= k) break;
                const int ii = (i0 + u) & 31;
                const double yi = __shfl_sync(0xffffffffu, z * dinv, ii);
                if (lane == ii) {
                    z = yi;
                    ys[i0 + u] = yi;
                }
                if (lane > ii) z = fma(-c[u], yi, z);
            }
        }
        sync();
        if (w > own) {
#pragma unroll
            for (int u = 0; u < kLuSub; ++u)
                if (i0 + u < k) z = fma(-c[u], ys[i0 + u], z);
        }
    }
    sync();  // ys is written again below
    load(nsub - 1);
    for (int sb = nsub - 1; sb >= 0; --sb) {
        const int i0 = kLuSub * sb, own = i0 >> 5;
#pragma unroll
        for (int u = 0; u < kLuSub; ++u) c[u] = cn[u];
        if (sb > 0) load(sb - 1);
        if (w == own) {
#pragma unroll
            for (int u = kLuSub - 1; u >= 0; --u) {
                if (i0 + u >= k) continue;
                const int ii = (i0 + u) & 31;
                const double xi = __shfl_sync(0xffffffffu, z, ii);
                if (lane == ii) ys[i0 + u] = xi;
                if (lane < ii) z = fma(-c[u], xi, z);
            }
        }
        sync();
        if (w < own) {
#pragma unroll
            for (int u = kLuSub - 1; u >= 0; --u)
                if (i0 + u < k) z = fma(-c[u], ys[i0 + u], z);
        }
    }
    return z;
}

}  // namespace cacg
