// Mixed-precision factorisation of one outer block [k0, k0+nb) (nb <= 128) of
// every large front of a level, once the block has received the updates of
// all earlier columns of its supernode:
//
//   k_diag_block   one CTA per front: A11 = L11 D L11^T in FP32 shared memory, a
//                  role per warp over 32-column sub-blocks (the chain of pivots,
//                  the elimination of the rows below and of the identity, which
//                  becomes X^T = L11^{-T}, the FP64 pivots, the updates).  Writes
//                  L11 and D to the factor, D and D^{-1} to a workspace slot, and
//                  X^T to the solves' inverse of the block (PanelTask::inv) or,
//                  where the solves' blocks are others, to the slot.  A block with
//                  a pivot that the chain does not decide is done again by
//                  diag_block_exact, pivot by pivot in FP64.
//   k_panel_solve  128 or 64 rows per CTA: W21 = A21 X^T as an FP32 register-tiled
//                  GEMM, L21 = W21 D^{-1}; L21 goes to the factor and, K-major,
//                  W21 and L21 go to the staging operands of the tensor-core
//                  updates.
//
// Together they replace the reference's per-column panel loop for these
// blocks (CAESolvers/UCHOL/UtduNumericFactorization.cs:520-610): the same
// L, D and pivot rule, computed in two launches per 128 columns instead of a
// chain of small steps.  The fronts of the mixed path are stored in FP32 and L,
// X and the products are FP32; the pivots are FP64: each diagonal entry of the
// block is carried in FP64 through every elimination step inside the block
// (d_r -= d_k L_rk^2 with the FP32 L), and the pivot test !(d > tol * scale),
// the regularisation and D itself are FP64 (the FP32 elimination divides by D
// rounded to FP32).  That is O(nb^2) FP64 work per block, done beside the chain of
// pivots, which runs on sums of two floats while every pivot is clearly decided.  The FP64 residual
// refinement recovers full accuracy of the solution.
#pragma once

#include <cfloat>
#include <climits>
#include <cuda_bf16.h>

#include "common.cuh"

namespace uchol_dev {

constexpr int kDiagMax = 128;
constexpr int kDiagLd = kDiagMax + 1;
// A block's inverse: X^T as kDiagMax x kDiagMax (row k, column j: X[j][k], zero for k > j and beyond nb), which is
// X column-major: the solves' inverse of the same block (PanelTask::inv), where there is one.  Workspace: a slot of D
// and D^{-1} (kDiagMax floats each) per block of the launch, then, where the solves have no such block, the inverses.
constexpr int kDiagSlotD = 2 * kDiagMax;
__host__ __device__ constexpr size_t minv_floats(size_t slots, bool with_inverses) {
    return slots * (kDiagSlotD + (with_inverses ? (size_t)kDiagMax * kDiagMax : 0));
}
__device__ __forceinline__ float* diag_slot_d(float* minv, const PanelTask& tk) {
    return minv + (size_t)tk.slot * (kDiagSlotD + (tk.inv < 0 ? kDiagMax * kDiagMax : 0));
}
template <class F>   // float or const float
__device__ __forceinline__ F* diag_slot_inverse(float* minv, F* linv, const PanelTask& tk) {
    return tk.inv < 0 ? diag_slot_d(minv, tk) + kDiagSlotD : linv + (size_t)tk.inv * kDiagMax * kDiagMax;
}
constexpr int kSolveRows = 128;
// float part: S and X (kDiagMax x kDiagLd each), Wt (kDiagMax x 33), D and D^{-1} in FP32;
// then the FP64 part: the running diagonal and D (kDiagMax doubles each)
constexpr size_t kDiagSmemFloats = 2 * kDiagMax * kDiagLd + kDiagMax * 33 + 2 * kDiagMax;
constexpr size_t kDiagExactBytes = sizeof(float) * kDiagSmemFloats + sizeof(double) * 2 * kDiagMax;
static_assert(sizeof(float) * kDiagSmemFloats % sizeof(double) == 0, "the FP64 part is aligned");

// Pivot acceptance of the reference, !(d > tol*scale) -> regularise or reject,
// on FP64 pivots (UtduNumericFactorization.cs:553-592).  Only the decision is
// taken per pivot; the smallest and largest |d| of the block are taken from D
// once it is complete (FP64 instructions are scarce on this GPU).
struct PivotAccD {
    int regularized = 0, negative = 0, failed = INT_MAX;
    __device__ __forceinline__ double accept(double piv, int column, double thr, double reg, int allow) {
        if (!(piv > thr)) {
            if (!allow) failed = min(failed, column);
            if (piv < 0.0) ++negative;
            ++regularized;
            piv = reg;
        }
        return piv;
    }
    __device__ __forceinline__ void flush(PivotStats* st) const {
        if (regularized) atomicAdd(&st->regularized, regularized);
        if (negative) atomicAdd(&st->negative, negative);
        if (failed != INT_MAX) atomicMin(&st->failed, failed);
    }
};

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// LDL^T of the bn x bn (bn <= 32) diagonal sub-block at S[b0][b0] by one
// warp, with the same eliminations applied to the identity so that
// X_bb = L_bb^{-1} comes out with it.  Lane r holds row b0 + r in registers
// as a shift register: at pivot k, a[j] is F[r][k + j] and x[c] is X[r][c];
// its diagonal entry is carried separately in FP64 (dd, from dg), and the pivot
// d_k is lane k's dd.
// Every lane below the pivot applies F[r][k+j] -= L[r][k] (d_k L[k+j][k])
// (the reference's association) and shifts its row by one, so the loop over
// pivots stays rolled (short code) while every register index is a constant.
// The pivot column (times d_k) and row k of X reach every lane through the
// 64-float shared scratch `scr` (16-byte aligned) as eight 16-byte broadcast
// loads each: lane r stores d_k L[r][k] at slot (r - k) mod 32, so slot j is
// row k + j (rows above the pivot store zero).  Entries right of the
// diagonal take meaningless updates and are never read.
__device__ __forceinline__ void warp_ldlt32(float* S, float* X, int b0, int bn, int lane, int col0, double thr,
                                            double reg, int allow, float* sd, float* sdi, double* dg, double* sd64,
                                            PivotAccD& acc, float* scr) {
    float a[32], x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        a[j] = (lane < bn && j <= lane) ? S[(b0 + lane) * kDiagLd + b0 + j] : 0.f;
        x[j] = j == lane ? 1.f : 0.f;
    }
    double dd = lane < bn ? dg[b0 + lane] : 0.0;   // this row's diagonal entry, FP64
    for (int k = 0; k < bn; ++k) {
        const double raw = __shfl_sync(0xffffffffu, dd, k);   // F[k][k]
        const double piv64 = acc.accept(raw, col0 + k, thr, reg, allow);   // the same in every lane
        const float piv = (float)piv64;
        const float inv = rcp_approx(piv);
        const bool below = lane > k && lane < bn;
        const float l = below ? a[0] * inv : 0.f;
        if (below) {
            S[(b0 + lane) * kDiagLd + b0 + k] = l;
            const double ld = (double)l;
            dd = fma(-piv64, ld * ld, dd);   // l^2 is exact in FP64
        }
        if (lane == k) {
            S[(b0 + k) * kDiagLd + b0 + k] = 1.f;
            sd[b0 + k] = piv;
            sdi[b0 + k] = inv;
            sd64[b0 + k] = piv64;
        }
        scr[(lane - k) & 31] = piv * l;
        if (lane == k) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                reinterpret_cast<float4*>(scr + 32)[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        }
        __syncwarp();
        float pl[32], xk[32];   // d_k L[k+j][k] (zero past the block), X[k][c]
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 u = reinterpret_cast<const float4*>(scr)[q];
            const float4 v = reinterpret_cast<const float4*>(scr + 32)[q];
            pl[4 * q] = u.x;
            pl[4 * q + 1] = u.y;
            pl[4 * q + 2] = u.z;
            pl[4 * q + 3] = u.w;
            xk[4 * q] = v.x;
            xk[4 * q + 1] = v.y;
            xk[4 * q + 2] = v.z;
            xk[4 * q + 3] = v.w;
        }
        __syncwarp();   // the scratch is rewritten at the next pivot
#pragma unroll
        for (int j = 1; j < 32; ++j) a[j - 1] = fmaf(-l, pl[j], a[j]);
        a[31] = 0.f;
#pragma unroll
        for (int c = 0; c < 32; ++c) x[c] = fmaf(-l, xk[c], x[c]);
    }
    if (lane < bn) {
#pragma unroll
        for (int c = 0; c < 32; ++c)
            if (c <= lane) X[(b0 + lane) * kDiagLd + b0 + c] = x[c];
    }
}

// The outer block with every elimination step's pivot taken on the FP64 diagonal as it is reached:
// the form that k_diag_block falls back to.  Threads 0..255 of the CTA; `sync` is their barrier.
__device__ __forceinline__ void diag_sync256() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __noinline__ void diag_block_exact(const PanelTask& tk, const SnDev& d, float* smem, float* __restrict__ panel,
                                              double* __restrict__ diag, float* __restrict__ M, float* __restrict__ Md,
                                              const FactorCtl& ctl, PivotStats* st) {
    float* S = smem;                         // block, row-major (S[r * kDiagLd + c]); L11 after the factorisation
    float* X = S + kDiagMax * kDiagLd;       // L11^{-1}, row-major
    float* Wt = X + kDiagMax * kDiagLd;      // W = L D of the current sub-block's rows below it
    float* sd = Wt + kDiagMax * 33;          // D
    float* sdi = sd + kDiagMax;              // D^{-1}
    double* dg = reinterpret_cast<double*>(smem + kDiagSmemFloats);   // running diagonal, FP64
    double* sd64 = dg + kDiagMax;            // D, FP64
    const double thr = ctl.threshold, reg = ctl.regularization;
    const int nb = tk.nb, k0 = tk.j0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* P = panel + d.panel_off + k0 + (long long)k0 * d.ldp;   // A11 origin, column-major, ld = ldp

    for (int i = tid; i < kDiagMax * kDiagLd; i += 256) X[i] = 0.f;
    // lower triangle of A11: 16 independent loads in flight per thread
    for (int q0 = 0; q0 < kDiagMax * kDiagMax / 256; q0 += 16) {
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int idx = tid + 256 * (q0 + q), r = idx & (kDiagMax - 1), c = idx >> 7;
            v[q] = (r < nb && c <= r) ? P[r + (long long)c * d.ldp] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int idx = tid + 256 * (q0 + q), r = idx & (kDiagMax - 1), c = idx >> 7;
            S[r * kDiagLd + c] = v[q];
        }
    }
    if (tid < kDiagMax) dg[tid] = tid < nb ? (double)P[tid + (long long)tid * d.ldp] : 0.0;
    diag_sync256();

    PivotAccD acc;
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const int bn = min(32, nb - b0);
        // (1) LDL^T of the sub-block and X_bb = L_bb^{-1}, by one warp
        if (warp == 0)   // Wt is free until step (3): its first 64 floats are the warp's scratch
            warp_ldlt32(S, X, b0, bn, lane, d.first_col + k0 + b0, thr, reg, ctl.allow_regularization, sd, sdi, dg,
                        sd64, acc, Wt);
        diag_sync256();
        // (3) rows below the sub-block: w[r][j] = sum_{k<=j} A[r][b0+k] X_bb[j][k], l = w / d_j;
        //     lane j, rows r0 + 8 q (four independent sums per lane)
        const int rb0 = b0 + bn;
        for (int r0 = rb0 + warp; r0 < nb; r0 += 32) {
            float w[4] = {0.f, 0.f, 0.f, 0.f};
            if (lane < bn) {
#pragma unroll 4
                for (int k = 0; k < bn; ++k) {
                    const float x = X[(b0 + lane) * kDiagLd + b0 + k];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int r = min(r0 + 8 * q, nb - 1);
                        w[q] = fmaf(S[r * kDiagLd + b0 + k], x, w[q]);
                    }
                }
            }
            __syncwarp();
            if (lane < bn) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = r0 + 8 * q;
                    if (r < nb) {
                        Wt[r * 33 + lane] = w[q];
                        S[r * kDiagLd + b0 + lane] = w[q] * sdi[b0 + lane];
                    }
                }
            }
        }
        diag_sync256();
        // (3b) the diagonal entries of the rows below, in FP64: d_r -= sum_k d_k L_rk^2, two threads per
        //      row (16 of the sub-block's columns each, four independent sums); reads only the
        //      sub-block's columns of S, which step (4) does not write
        {
            const int r = rb0 + (tid >> 1), kh = (tid & 1) * 16;
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            if (r < nb) {
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    if (kh + k < bn) {
                        const double l = (double)S[r * kDiagLd + b0 + kh + k];
                        v[k & 3] = fma(sd64[b0 + kh + k], l * l, v[k & 3]);
                    }
                }
            }
            double sum = (v[0] + v[1]) + (v[2] + v[3]);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            if (r < nb && kh == 0) dg[r] -= sum;
        }
        // (4) trailing update of the block: S[r][c] -= sum_k W[r][k] L[c][k], rb0 <= c <= r < nb
        if (rb0 < nb) {
            const int tx = tid & 15, ty = tid >> 4;
            float accu[6][6];
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int q = 0; q < 6; ++q) accu[p][q] = 0.f;
#pragma unroll 2
            for (int k = 0; k < bn; ++k) {
                float wv[6], lv[6];
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    const int r = rb0 + ty + 16 * p;
                    wv[p] = r < nb ? Wt[r * 33 + k] : 0.f;
                }
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const int c = rb0 + tx + 16 * q;
                    lv[q] = c < nb ? S[c * kDiagLd + b0 + k] : 0.f;
                }
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int q = 0; q < 6; ++q) accu[p][q] = fmaf(wv[p], lv[q], accu[p][q]);
            }
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const int r = rb0 + ty + 16 * p, c = rb0 + tx + 16 * q;
                    if (r < nb && c <= r) S[r * kDiagLd + c] -= accu[p][q];
                }
        }
        diag_sync256();
    }

    // (5) off-diagonal blocks of X = L11^{-1}: X_ij = -X_ii sum_{j<=k<i} L_ik X_kj, by block diagonals;
    //     64 threads per block pair, each a 4 x 4 tile (rows rr + 8q, columns cc + 8p)
    const int nblk = (nb + 31) >> 5;
    float* T = Wt;   // (nblk - dd) blocks of 32 x 33
    for (int dd = 1; dd < nblk; ++dd) {
        const int pairs = nblk - dd;
        const int pr = tid >> 6, cc = tid & 7, rr = (tid >> 3) & 7, i = pr + dd;
        const bool active = pr < pairs;
        float t[4][4];
        if (active) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int p = 0; p < 4; ++p) t[q][p] = 0.f;
#pragma unroll 2
            for (int k = pr * 32; k < i * 32; ++k) {
                float xv[4], sv[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) xv[p] = X[k * kDiagLd + pr * 32 + cc + 8 * p];
#pragma unroll
                for (int q = 0; q < 4; ++q) sv[q] = S[(i * 32 + rr + 8 * q) * kDiagLd + k];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int p = 0; p < 4; ++p) t[q][p] = fmaf(sv[q], xv[p], t[q][p]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int p = 0; p < 4; ++p) T[pr * 32 * 33 + (rr + 8 * q) * 33 + cc + 8 * p] = t[q][p];
        }
        diag_sync256();
        if (active) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int p = 0; p < 4; ++p) t[q][p] = 0.f;
            // X_ii is lower triangular (zero above its diagonal), so the sums run over all 32 columns
#pragma unroll 2
            for (int tt = 0; tt < 32; ++tt) {
                float yv[4], xv[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) yv[p] = T[pr * 32 * 33 + tt * 33 + cc + 8 * p];
#pragma unroll
                for (int q = 0; q < 4; ++q) xv[q] = X[(i * 32 + rr + 8 * q) * kDiagLd + i * 32 + tt];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int p = 0; p < 4; ++p) t[q][p] = fmaf(xv[q], yv[p], t[q][p]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int row = i * 32 + rr + 8 * q;
                if (row < nb) {
#pragma unroll
                    for (int p = 0; p < 4; ++p) X[row * kDiagLd + pr * 32 + cc + 8 * p] = -t[q][p];
                }
            }
        }
        diag_sync256();
    }

    // (6) write L11 (unit diagonal), D, and the workspace slot
    for (int c = warp; c < nb; c += 8)
        for (int r = c + lane; r < nb; r += 32) P[r + (long long)c * d.ldp] = r == c ? 1.f : S[r * kDiagLd + c];
    if (tid < nb) diag[d.first_col + k0 + tid] = sd64[tid];
    for (int idx = tid; idx < kDiagMax * kDiagMax; idx += 256) {
        const int k = idx >> 7, j = idx & (kDiagMax - 1);
        M[idx] = (j < nb && k <= j) ? X[j * kDiagLd + k] : 0.f;
    }
    if (tid < kDiagMax) {
        Md[tid] = tid < nb ? sd[tid] : 0.f;
        Md[kDiagMax + tid] = tid < nb ? sdi[tid] : 0.f;
    }
    if (tid == 0) acc.flush(st);
    // smallest and largest |d| of the block, by the first warp
    if (warp == 0) {
        double lo = DBL_MAX, hi = 0.0;
        for (int k = lane; k < nb; k += 32) {
            const double a = fabs(sd64[k]);
            lo = fmin(lo, a);
            hi = fmax(hi, a);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0 && nb > 0) {
            atomicMin(&st->min_bits, (unsigned long long)__double_as_longlong(lo));
            atomicMax(&st->max_bits, (unsigned long long)__double_as_longlong(hi));
        }
    }
}

// ---- k_diag_block: the outer block by one CTA of kDiagThreads threads with a role per warp.
//
// What bounds it: a chain of nb pivots on one SM, each needing the one before it.  FP64 instructions take 64
// cycles each here (issue and latency, however few lanes are active), so a pivot taken wholly in FP64 costs six
// of them; the chain therefore carries each row's diagonal as an unevaluated sum of two floats (df_sub: about
// 48 bits, 12 dependent FP32 operations), and the FP64 diagonal D itself is accumulated beside it by three other
// warps from the same FP32 L (the same sums d_r -= d_k l_rk^2).  The eliminations of the rows below the
// sub-block and of the identity (which become X^T) follow the chain eight pivots behind in four warps, and the
// rank-32 updates of the columns beyond the next sub-block run beside the next sub-block's chain.
//   chain   (1 warp)   LDL^T of the 32 x 32 diagonal sub-block, lane = row
//   rows    (4 warps)  lane = row: W = A L^-T of the rows below the sub-block, L = W / D, and the same
//                      elimination of the identity's rows up to the sub-block, which gives X^T (128 rows in all)
//   fp64    (3 warps)  D: the sub-block's own recursion, then its part of the later rows' diagonals
//   update  (4 warps)  W L^T of later columns (of the next sub-block's columns together with the rows warps)
// The chain shares its scheduler (warp number mod 4) with two FP64 warps only, which issue little.
//
// A pivot whose two-float value is not clearly above the rejection threshold, or that lost more than 20 bits of
// its diagonal entry, or that leaves the range in which the low words are normal floats, is not decided here:
// the whole block is factorised again by diag_block_exact (nothing has been written to the factor by then).
constexpr int kDiagThreads = 384;
constexpr int kDiagRowLd = 132;             // S[c * kDiagRowLd + r]: 16-byte aligned columns, conflict-free rows
constexpr float kDiagKeep = 0x1p-20f;       // smallest pivot / diagonal entry taken by the fast chain
// floats: S (128 x 132), W (2 x 32 x 132), per-pivot {D hi, D lo, 1/D, -} (128 x 4), pivot column (2 x 64),
// running diagonal of every row and its limit (3 x 128); then FP64: running diagonal, D (128 each), partial sums (32)
constexpr size_t kDiagFastFloats = (size_t)kDiagMax * kDiagRowLd + 2 * 32 * kDiagRowLd + 4 * kDiagMax + 128 + 3 * kDiagMax;
constexpr size_t kDiagFastBytes = sizeof(float) * kDiagFastFloats + sizeof(double) * (2 * kDiagMax + 32);
static_assert(sizeof(float) * kDiagFastFloats % 16 == 0, "the FP64 part is aligned");
constexpr size_t kDiagSmemBytes = kDiagFastBytes > kDiagExactBytes ? kDiagFastBytes : kDiagExactBytes;

// (h, l) -= (d, dl) x^2 on unevaluated two-float sums; x^2 and d x^2 are formed exactly (product and remainder).
__device__ __forceinline__ void df_sub(float& h, float& l, float d, float dl, float x) {
    const float p = __fmul_rn(x, x), pl = __fmaf_rn(x, x, -p);
    const float q = __fmul_rn(d, p);
    const float ql = __fmaf_rn(dl, p, __fmaf_rn(d, pl, __fmaf_rn(d, p, -q)));
    const float s = __fsub_rn(h, q), bb = __fsub_rn(s, h);
    const float err = __fsub_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fadd_rn(q, bb));
    const float lo = __fsub_rn(__fadd_rn(l, err), ql);
    h = __fadd_rn(s, lo);
    l = __fsub_rn(lo, __fsub_rn(h, s));
}

// x^2 as a double, exactly, without FP64 instructions: the 48-bit product of the significands under the
// doubled exponent (subnormal x counts as zero).
__device__ __forceinline__ double exact_square(float x) {
    const unsigned u = __float_as_uint(x), e = (u >> 23) & 255u;
    const unsigned m = (u & 0x7fffffu) | 0x800000u;
    const unsigned long long mm = (unsigned long long)m * m;   // [2^46, 2^48)
    const unsigned top = (unsigned)(mm >> 47);
    const unsigned long long bits = (mm << (6 - top)) + ((unsigned long long)(2 * e + 768 + top) << 52);
    return e == 0 ? 0.0 : __longlong_as_double((long long)bits);
}

// Two FP32 multiply-adds in one instruction (the FP32 pipe's rate is the same; the issue slots saved go to the
// shared-memory loads beside them).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <int kId, int kCount>
__device__ __forceinline__ void diag_bar_sync() { asm volatile("bar.sync %0, %1;" ::"n"(kId), "n"(kCount) : "memory"); }
__device__ __forceinline__ void diag_bar_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void diag_bar_arrive(int id, int count) {
    __threadfence_block();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// S[c][r] -= sum_k W[k][r] L[k][c] (L[k][c] = S[b0 + k][c]) for the NR x NC block at (r0, c0) by one warp:
// lane tile of NR / 4 rows (groups of four, 16 apart) by NC / 8 columns.  Shared-memory bandwidth bounds it (a
// 16-byte load occupies the SM's load path for four cycles), so the 32 x 32 block's lane tile is 8 x 4.
template <int NR, int NC>
__device__ __forceinline__ void diag_update_block(float* S, const float* W, int b0, int r0, int c0, int lane) {
    constexpr int G = NR / 16, CL = NC / 8;
    const int r = r0 + 4 * (lane & 3), c = c0 + CL * (lane >> 2);
    f32x2 acc[CL][2 * G];
#pragma unroll
    for (int q = 0; q < CL; ++q)
#pragma unroll
        for (int p = 0; p < 2 * G; ++p) acc[q][p] = 0ull;
    const float* wp = W + r;
    const float* lp = S + b0 * kDiagRowLd + c;
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        f32x2 w[2 * G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(wp + k * kDiagRowLd + 16 * g);
            w[2 * g] = v.x;
            w[2 * g + 1] = v.y;
        }
        float l[CL];
        if constexpr (CL == 4) {
            const float4 v = *reinterpret_cast<const float4*>(lp + k * kDiagRowLd);
            l[0] = v.x;
            l[1] = v.y;
            l[2] = v.z;
            l[3] = v.w;
        } else {
            const float2 v = *reinterpret_cast<const float2*>(lp + k * kDiagRowLd);
            l[0] = v.x;
            l[1] = v.y;
        }
#pragma unroll
        for (int q = 0; q < CL; ++q)
#pragma unroll
            for (int p = 0; p < 2 * G; ++p) acc[q][p] = fma2(w[p], pack2(l[q], l[q]), acc[q][p]);
    }
#pragma unroll
    for (int q = 0; q < CL; ++q)
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float4* o = reinterpret_cast<float4*>(S + (c + q) * kDiagRowLd + r + 16 * g);
            float4 v = *o;
            float x[4];
            unpack2(acc[q][2 * g], x[0], x[1]);
            unpack2(acc[q][2 * g + 1], x[2], x[3]);
            v.x -= x[0];
            v.y -= x[1];
            v.z -= x[2];
            v.w -= x[3];
            *o = v;
        }
}

__device__ __forceinline__ float diag_entry(const f32x2 (&a)[16], int j) {   // j: compile-time
    float x, y;
    unpack2(a[j >> 1], x, y);
    return (j & 1) ? y : x;
}

struct DiagShared {
    float *S, *W, *scr, *rh, *rl, *lim;
    float4* piv;
    double *dg, *sd64, *part;
};

// The chain's state (lane = row of the sub-block).
struct DiagChain {
    f32x2 a[16];      // this row's entries of columns 4 g + j, two a register pair (shifted down after each quad)
    float h, l;       // the row's running diagonal
    float least;
    bool good;
};
// Pivots 4 g .. 4 g + 3 of the chain, NP register pairs of columns (those past the sub-block's end carry nothing).
// Only the next pivot's column is updated at once; the other columns' updates wait until the next pivot, in the
// shadow of its reciprocal.  Short loops over quads: unrolled further, instruction fetches bound the chain.
// a[p] += m * v[p] for the register pairs p in [P0, P1).
template <int P0, int P1>
__device__ __forceinline__ void diag_axpy(f32x2 (&a)[16], f32x2 m, const ulonglong2 (&v)[8]) {
#pragma unroll
    for (int p = P0; p < P1; ++p) a[p] = fma2(m, (p & 1) ? v[p >> 1].y : v[p >> 1].x, a[p]);
}
template <int NP, int KK>
__device__ __forceinline__ void diag_pivot(const DiagShared& X, DiagChain& C, ulonglong2 (&v)[8], f32x2& m, int b0, int g,
                                           int lane) {
    constexpr int kNext = (KK + 1) / 2;        // pair that holds column KK + 1
    const int k = 4 * g + KK;
    float* sc = X.scr + 64 * (KK & 1);         // two buffers: one warp barrier per pivot
    const float ph = __shfl_sync(0xffffffffu, C.h, k), pl = __shfl_sync(0xffffffffu, C.l, k);
    const float ak = diag_entry(C.a, KK);
    sc[lane] = ak;
    const float inv = rcp_approx(ph);
    if constexpr (KK > 0) diag_axpy<KK / 2 + 1, NP>(C.a, m, v);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NP / 2; ++q) v[q] = reinterpret_cast<const ulonglong2*>(sc + 4 * g)[q];
    const float lk = lane > k ? ak * inv : 0.f;
    m = pack2(-lk, -lk);
    diag_axpy<kNext, (KK == 3 ? NP : kNext + 1)>(C.a, m, v);
    df_sub(C.h, C.l, ph, pl, lk);
    X.S[(b0 + k) * kDiagRowLd + b0 + lane] = lk;
    if (lane == k) X.piv[b0 + k] = make_float4(ph, pl, inv, 0.f);
    C.good = lane == k ? ph > C.least && ph < 1e30f : C.good;
}
template <int NP>
__device__ __forceinline__ void diag_quad(const DiagShared& X, DiagChain& C, int b0, int g, int lane) {
    ulonglong2 v[8];   // the pivot's column (W)
    f32x2 m = 0ull;    // -L of this row
    diag_pivot<NP, 0>(X, C, v, m, b0, g, lane);
    diag_pivot<NP, 1>(X, C, v, m, b0, g, lane);
    diag_pivot<NP, 2>(X, C, v, m, b0, g, lane);
    diag_pivot<NP, 3>(X, C, v, m, b0, g, lane);
    __syncwarp();
    if (g & 1) diag_bar_arrive(2 + (g >> 1), 192);   // eight more columns of L are in S
#pragma unroll
    for (int j = 0; j < NP - 2; ++j) C.a[j] = C.a[j + 2];
}

// The chain over sub-block b0: L into S, pivots into piv; columns are published to the rows and FP64 warps in eights
// (barriers 2 .. 5).  Returns whether every pivot could be decided.
__device__ __forceinline__ bool diag_chain(const DiagShared& X, int b0, int lane) {
    DiagChain C;
#pragma unroll
    for (int j = 0; j < 16; ++j) {   // entries from the diagonal on are not the chain's
        const float x = X.S[(b0 + 2 * j) * kDiagRowLd + b0 + lane], y = X.S[(b0 + 2 * j + 1) * kDiagRowLd + b0 + lane];
        C.a[j] = pack2(2 * j < lane ? x : 0.f, 2 * j + 1 < lane ? y : 0.f);
    }
    C.h = X.rh[b0 + lane];
    C.l = X.rl[b0 + lane];
    C.least = X.lim[b0 + lane];
    C.good = true;
#pragma unroll 1
    for (int g = 0; g < 4; ++g) diag_quad<16>(X, C, b0, g, lane);
#pragma unroll 1
    for (int g = 4; g < 8; ++g) diag_quad<8>(X, C, b0, g, lane);
    return C.good;
}

// Row r = 32 rw + lane against sub-block b0: see k_diag_block.
struct DiagRows {
    f32x2 a[16];
    float h, l;
    int r;
    bool below;   // the same in a warp
};
template <int NP, int KK>
__device__ __forceinline__ void diag_rows_pivot(const DiagShared& X, DiagRows& R, float* W, int b0, int g) {
    const int k = 4 * g + KK;
    const float4 pv = X.piv[b0 + k];
    ulonglong2 v[8];   // L of this pivot, zero up to its row
#pragma unroll
    for (int q = 0; q < NP / 2; ++q)
        v[q] = reinterpret_cast<const ulonglong2*>(X.S + (b0 + k) * kDiagRowLd + b0 + 4 * g)[q];
    const float w = diag_entry(R.a, KK);
    diag_axpy<(KK + 1) / 2, NP>(R.a, pack2(-w, -w), v);
    W[k * kDiagRowLd + R.r] = w;
    const float lr = w * pv.z;
    if (R.below) X.S[(b0 + k) * kDiagRowLd + R.r] = lr;
    df_sub(R.h, R.l, pv.x, pv.y, lr);   // (of no use for the identity's rows)
}
template <int NP>
__device__ __forceinline__ void diag_rows_quad(const DiagShared& X, DiagRows& R, float* W, float* M, int b0, int g, int nb) {
    if (!(g & 1)) diag_bar_sync(2 + (g >> 1), 192);
    diag_rows_pivot<NP, 0>(X, R, W, b0, g);
    diag_rows_pivot<NP, 1>(X, R, W, b0, g);
    diag_rows_pivot<NP, 2>(X, R, W, b0, g);
    diag_rows_pivot<NP, 3>(X, R, W, b0, g);
    // X^T of these columns: zero for the rows below, and past the block
    float y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = !R.below && R.r < nb && b0 + 4 * g + q < nb ? diag_entry(R.a, q) : 0.f;
    *reinterpret_cast<float4*>(M + R.r * kDiagMax + b0 + 4 * g) = make_float4(y[0], y[1], y[2], y[3]);
#pragma unroll
    for (int j = 0; j < NP - 2; ++j) R.a[j] = R.a[j + 2];
}
__device__ __forceinline__ void diag_rows(const DiagShared& X, float* W, float* M, int b0, int rw, int lane, int nb) {
    DiagRows R;
    const int r = 32 * rw + lane;
    const bool own = 32 * rw == b0;
    R.r = r;
    R.below = 32 * rw > b0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float x = X.S[(b0 + 2 * j) * kDiagRowLd + r], y = X.S[(b0 + 2 * j + 1) * kDiagRowLd + r];
        R.a[j] = pack2(own ? (2 * j == lane ? 1.f : 0.f) : x, own ? (2 * j + 1 == lane ? 1.f : 0.f) : y);
    }
    R.h = X.rh[r];
    R.l = X.rl[r];
#pragma unroll 1
    for (int g = 0; g < 4; ++g) diag_rows_quad<16>(X, R, W, M, b0, g, nb);
#pragma unroll 1
    for (int g = 4; g < 8; ++g) diag_rows_quad<8>(X, R, W, M, b0, g, nb);
    if (R.below) {
        X.rh[r] = R.h;
        X.rl[r] = R.l;
    }
}

// Sum of d_k l_rk^2 over pivots k0 .. k0 + n - 1 taken off dd (row r).
__device__ __forceinline__ double diag_fp64_part(const DiagShared& X, int k0, int n, int r, double dd) {
#pragma unroll 8
    for (int k = 0; k < n; ++k) dd = fma(-X.sd64[k0 + k], exact_square(X.S[(k0 + k) * kDiagRowLd + r]), dd);
    return dd;
}

// D in FP64 beside the chain: warp q = 0 follows it with the sub-block's recursion, then shares the next sub-block's
// rows with warp 1 (half of the pivots each); warps 2 and 1 take the rows after those.
__device__ __forceinline__ void diag_fp64(const DiagShared& X, int nblk, int q, int lane) {
    double next = q == 0 ? X.dg[lane] : 0.0;
    for (int b = 0; b < nblk; ++b) {
        const int b0 = 32 * b, r1 = b0 + 32 + lane;
        if (q == 0) {
            double dd = next;
#pragma unroll 1
            for (int g = 0; g < 8; ++g) {
                if (!(g & 1)) diag_bar_sync(2 + (g >> 1), 192);
                double sq[4];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) sq[kk] = exact_square(X.S[(b0 + 4 * g + kk) * kDiagRowLd + b0 + lane]);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {   // zero squares up to the pivot's row
                    const double dk = __shfl_sync(0xffffffffu, dd, 4 * g + kk);
                    dd = fma(-dk, sq[kk], dd);
                }
            }
            X.sd64[b0 + lane] = dd;
        }
        diag_bar_sync(12 + b, kDiagThreads);   // the sub-block's L is complete, and its D
        if (b + 1 >= nblk) break;
        if (q == 0) {
            next = diag_fp64_part(X, b0, 16, r1, X.dg[r1]);
            diag_bar_sync<10, 64>();
            next += X.part[lane];
        } else if (q == 1) {
            X.part[lane] = diag_fp64_part(X, b0 + 16, 16, r1, 0.0);
            diag_bar_sync<10, 64>();
        }
        const int rb = q == 2 ? b + 2 : q == 1 ? b + 3 : nblk;
        if (rb < nblk) X.dg[32 * rb + lane] = diag_fp64_part(X, b0, 32, 32 * rb + lane, X.dg[32 * rb + lane]);
    }
}

__global__ void __launch_bounds__(kDiagThreads, 1) k_diag_block(const PanelTask* __restrict__ tasks, const SnDev* __restrict__ sn,
                                                             float* __restrict__ panel, double* __restrict__ diag,
                                                             float* __restrict__ minv, float* __restrict__ linv,
                                                             const FactorCtl* __restrict__ ctlp, PivotStats* st) {
    extern __shared__ __align__(16) float smem[];
    DiagShared X;
    X.S = smem;                                     // column c, row r at S[c * kDiagRowLd + r]; L as the columns finish
    X.W = X.S + kDiagMax * kDiagRowLd;              // W of two sub-blocks, [k][row]
    X.piv = reinterpret_cast<float4*>(X.W + 2 * 32 * kDiagRowLd);   // per pivot: D (two floats), 1/D
    X.scr = reinterpret_cast<float*>(X.piv + kDiagMax);             // the chain's pivot column, two buffers
    X.rh = X.scr + 128;                             // running diagonal of every row, two floats
    X.rl = X.rh + kDiagMax;
    X.lim = X.rl + kDiagMax;                        // smallest pivot the chain decides, per row
    X.dg = reinterpret_cast<double*>(smem + kDiagFastFloats);       // running diagonal, FP64
    X.sd64 = X.dg + kDiagMax;                       // D, FP64
    X.part = X.sd64 + kDiagMax;
    __shared__ int bad;
    const PanelTask tk = tasks[blockIdx.x];
    const SnDev d = sn[tk.s];
    const FactorCtl ctl = *ctlp;
    const int nb = tk.nb, k0 = tk.j0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* S = X.S;
    float* P = panel + d.panel_off + k0 + (long long)k0 * d.ldp;   // A11 origin, column-major, ld = ldp
    float* Md = diag_slot_d(minv, tk);
    float* M = diag_slot_inverse(minv, linv, tk);

    // lower triangle into S, 16 bytes at a time (zero above the diagonal's group of four and past nb rows)
    for (int q = tid; q < kDiagMax * (kDiagMax / 4); q += kDiagThreads) {
        const int c = q >> 5, r = (q & 31) * 4;
        const int left = r + 3 < c || c >= nb ? 0 : min(4, max(0, nb - r));
        const float* src = left > 0 ? P + r + (long long)c * d.ldp : P;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(S + c * kDiagRowLd + r)),
                     "l"(src), "r"(4 * left)
                     : "memory");
    }
    if (tid == 0) bad = 0;
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (tid < kDiagMax) {
        if (tid >= nb) S[tid * kDiagRowLd + tid] = 1.f;   // rows past the block: identity, of no effect
        const float a = S[tid * kDiagRowLd + tid];
        X.rh[tid] = a;
        X.rl[tid] = 0.f;
        X.lim[tid] = tid < nb ? fmaxf(fmaxf(4.f * (float)ctl.threshold, 1e-25f), kDiagKeep * a) : 0.f;
        X.dg[tid] = (double)a;
    }
    __syncthreads();

    const int nblk = (nb + 31) >> 5;
    // warp -> role: 0 chain; 1, 2, 3, 5 rows; 9, 8, 4 FP64; 6, 7, 10, 11 update
    const int fp64 = warp == 9 ? 0 : warp == 8 ? 1 : warp == 4 ? 2 : -1;
    const int rows = warp < 4 ? warp - 1 : warp == 5 ? 3 : -1;
    // Each role runs its own loop over the sub-blocks (short jumps: a trip through shared code costs instruction
    // fetches).  Barrier 1 ends a sub-block; barrier 11: the next diagonal sub-block is up to date.
    if (fp64 >= 0) {
        diag_fp64(X, nblk, fp64, lane);
    } else if (warp == 0) {
        bool good = true;
#pragma unroll 1
        for (int b = 0;; ++b) {
            good &= diag_chain(X, 32 * b, lane);
            if (!good) bad = 1;
            diag_bar_sync<1, 288>();
            diag_bar_arrive(12 + b, kDiagThreads);
            if (b + 1 == nblk) break;
            diag_bar_sync<11, 160>();
        }
    } else if (rows >= 0) {
#pragma unroll 1
        for (int b = 0;; ++b) {
            float* W = X.W + (b & 1) * 32 * kDiagRowLd;
            diag_rows(X, W, M, 32 * b, rows, lane, nb);
            diag_bar_sync<1, 288>();
            diag_bar_arrive(12 + b, kDiagThreads);
            if (b + 1 == nblk) break;
            // this warp's rows of the next sub-block's columns
            if (rows != b + 1 && rows < nblk) diag_update_block<32, 32>(S, W, 32 * b, 32 * rows, 32 * b + 32, lane);
            __syncwarp();
        }
    } else {
        const int upd = warp < 8 ? warp - 6 : warp - 8;
#pragma unroll 1
        for (int b = 0;; ++b) {
            diag_bar_sync<1, 288>();
            diag_bar_arrive(12 + b, kDiagThreads);
            if (b + 1 == nblk) break;
            const float* W = X.W + (b & 1) * 32 * kDiagRowLd;
            diag_update_block<16, 16>(S, W, 32 * b, 32 * b + 32 + 16 * (upd & 1), 32 * b + 32 + 16 * (upd >> 1), lane);
            diag_bar_sync<11, 160>();
            // the columns past the next sub-block, beside its chain
            int unit = 0;
            for (int c = b + 2; c < nblk; ++c)
                for (int r = 0; r < nblk; ++r)
                    if ((r <= b || r >= c) && (unit++ & 3) == upd)
                        diag_update_block<32, 32>(S, W, 32 * b, 32 * r, 32 * c, lane);
        }
    }
    __syncthreads();
    if (bad) {
        if (tid < 256) diag_block_exact(tk, d, smem, panel, diag, M, Md, ctl, st);
        return;
    }
    // L11 to the factor: a thread per column, one bulk copy of whole groups of four rows below the diagonal's group
    if (tid < nb) {
        const int c = tid, r0 = min(nb, (c + 4) & ~3), r1 = max(r0, nb & ~3);
        float* o = P + (long long)c * d.ldp;
        const float* x = S + c * kDiagRowLd;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (r1 > r0)
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\ncp.async.bulk.commit_group;" ::"l"(o + r0),
                         "r"((unsigned)__cvta_generic_to_shared(x + r0)), "r"(4 * (r1 - r0))
                         : "memory");
        o[c] = 1.f;
        for (int r = c + 1; r < r0; ++r) o[r] = x[r];
        for (int r = r1; r < nb; ++r) o[r] = x[r];
    }
    // D, the rest of the workspace slot (X^T past the last sub-block), the smallest and largest pivot
    if (tid < nb) diag[d.first_col + k0 + tid] = X.sd64[tid];
    if (tid < kDiagMax) {
        const float4 pv = tid < nb ? X.piv[tid] : make_float4(0.f, 0.f, 0.f, 0.f);
        Md[tid] = pv.x;
        Md[kDiagMax + tid] = pv.z;
    }
    for (int q = tid; q < kDiagMax * (kDiagMax - 32 * nblk); q += kDiagThreads) {
        const int wc = kDiagMax - 32 * nblk;
        M[q / wc * kDiagMax + 32 * nblk + q % wc] = 0.f;
    }
    if (warp == 11 && nb > 0) {
        unsigned long long lo = ~0ull, hi = 0;   // every pivot is positive: ordered as its bits
        for (int k = lane; k < nb; k += 32) {
            const unsigned long long v = (unsigned long long)__double_as_longlong(X.sd64[k]);
            lo = min(lo, v);
            hi = max(hi, v);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            atomicMin(&st->min_bits, lo);
            atomicMax(&st->max_bits, hi);
        }
    }
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the copies have read S
}

// 4-byte asynchronous copy global -> shared (zero fill when !valid: nothing is read then).
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 4 : 0)
                 : "memory");
}
// 16-byte asynchronous copy global -> shared of the first `bytes` bytes (zero fill after them).
__device__ __forceinline__ void cp_async16z(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Shared memory of k_panel_solve: stages of (A21 chunk, X^T chunk), 32 K columns each; two for tiles of 128 rows, all four
// for tiles of 64.
constexpr int kPanelKc = 32;
template <int ROWS>
constexpr int kPanelStages = ROWS == 64 ? 4 : 2;
template <int ROWS>
constexpr int kPanelStageFloats = kPanelKc * (ROWS + 4 + kDiagMax + 4);
template <int ROWS>
constexpr size_t panel_smem_bytes() { return sizeof(float) * kPanelStages<ROWS> * kPanelStageFloats<ROWS>; }
static_assert(kPanelStages<128> * kPanelStageFloats<128> >= kDiagMax * 132 &&
              kPanelStages<64> * kPanelStageFloats<64> >= kDiagMax * 68,
              "the stages hold the tile of L21 on its way to the factor");

__device__ __forceinline__ void store_op4(__nv_bfloat16* p, float a, float b, float c, float e) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, e);
    uint2 v;
    v.x = *reinterpret_cast<unsigned*>(&lo);
    v.y = *reinterpret_cast<unsigned*>(&hi);
    *reinterpret_cast<uint2*>(p) = v;
}
// TF32 operands: rounded to TF32 precision (nearest, ties away) as they are staged, so that
// the tensor core, which reads only the top 19 bits of each FP32 operand, multiplies rounded
// rather than truncated values (truncation biases every product the same way, and over the
// many updates of a deep tree that bias accumulates in the factor).
__device__ __forceinline__ float round_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}
__device__ __forceinline__ void store_op4(float* p, float a, float b, float c, float e) {
    *reinterpret_cast<float4*>(p) = make_float4(round_tf32(a), round_tf32(b), round_tf32(c), round_tf32(e));
}
__device__ __forceinline__ void store_op1(__nv_bfloat16* p, float a) { *p = __float2bfloat16_rn(a); }
__device__ __forceinline__ void store_op1(float* p, float a) { *p = a; }

// W21 = A21 X^T and L21 = W21 D^{-1} for rows [row0, row0 + rows) of the
// front, 2 ROWS threads: thread (ty, tx) owns rows {4ty..4ty+3, ROWS/2+4ty..} and
// columns {4tx..4tx+3, 64+4tx..} of the ROWS x 128 tile (conflict-free 128-bit
// shared loads; two rows per FP32 instruction).  X^T is upper triangular, so
// columns below 64 take no updates from K >= 64.  L21 goes to the factor through
// shared memory, so that a column's rows are written together.  The SM's FP32 pipe
// (6 us a tile) and the launch bound it: 11,000 rows, 25.9 us with 4-byte
// copies and stores of 16 scattered bytes a thread, 22.5 us now (timed alone).
// Launches of fewer rows take tiles of 64, half the pipe's time, with all of
// their copies in flight at once (panel_rows in plan.cpp).
template <class Op, int ROWS>
__global__ void __launch_bounds__(2 * ROWS, 2) k_panel_solve(const PanelTask* __restrict__ tasks,
                                                     const SnDev* __restrict__ sn, float* __restrict__ panel,
                                                     float* __restrict__ minv, const float* __restrict__ linv,
                                                     Op* __restrict__ stage_a, Op* __restrict__ stage_b,
                                                     const StageInfo* __restrict__ stage_info) {
    constexpr int KC = kPanelKc, NT = 2 * ROWS, LDS = ROWS + 4, LDM = kDiagMax + 4;
    constexpr int NS = kPanelStages<ROWS>, SF = kPanelStageFloats<ROWS>;
    extern __shared__ __align__(16) float psm[];   // stage s: As = psm + s SF, Ms = As + KC LDS
    const PanelTask tk = tasks[blockIdx.x];
    const SnDev d = sn[tk.s];
    const int nb = tk.nb, k0 = tk.j0, row0 = tk.row0, rows = tk.rows;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const float* M = diag_slot_inverse<const float>(minv, linv, tk);
    float* A = panel + d.panel_off + row0 + (long long)k0 * d.ldp;   // A21 rows of this task, column-major
    f32x2 acc2[2][2][8];   // [row group][pair of rows][column]
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc2[i][0][j] = acc2[i][1][j] = 0ull;
    // K chunks of KC columns copied asynchronously into NS stages: every copy of a chunk in
    // flight at once, and the next NS - 1 chunks' copies under the current chunk's products
    const bool aligned = ((row0 | (int)(d.panel_off & 3)) & 3) == 0;   // rows on 16-byte boundaries
    auto issue_chunk = [&](int kc, int st) {
        float* As = psm + st * SF;
        float* Ms = As + KC * LDS;
        if (aligned) {
#pragma unroll
            for (int q = 0; q < (KC * ROWS) / (4 * NT); ++q) {
                const int idx = tid + NT * q, r = (idx % (ROWS / 4)) * 4, k = idx / (ROWS / 4);
                const int left = kc + k < nb ? min(4, max(0, rows - r)) : 0;
                cp_async16z(&As[k * LDS + r], left > 0 ? A + r + (long long)(kc + k) * d.ldp : A, 4 * left);
            }
        } else {
#pragma unroll
            for (int q = 0; q < (KC * ROWS) / NT; ++q) {
                const int idx = tid + NT * q, r = idx % ROWS, k = idx / ROWS;
                const bool ok = r < rows && kc + k < nb;
                cp_async4(&As[k * LDS + r], ok ? A + r + (long long)(kc + k) * d.ldp : A, ok);
            }
        }
#pragma unroll
        for (int q = 0; q < (KC * kDiagMax) / (4 * NT); ++q) {
            const int idx = tid + NT * q, r = (idx & 31) * 4, k = idx >> 5;
            cp_async16z(&Ms[k * LDM + r], M + (kc + k) * kDiagMax + r, 16);
        }
        cp_async_commit();
    };
    const int nch = (nb + KC - 1) / KC;
    for (int c = 0; c < min(NS - 1, nch); ++c) issue_chunk(c * KC, c);
    for (int c = 0; c < nch; ++c) {
        if (c + NS - 1 < nch) issue_chunk((c + NS - 1) * KC, (c + NS - 1) % NS);
        const int later = min(NS - 1, nch - 1 - c);   // chunks in flight after this one
        if (later >= 3) cp_async_wait<3>();
        else if (later == 2) cp_async_wait<2>();
        else if (later == 1) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        const int kc = c * KC;
        const float* As = psm + (c % NS) * SF;
        const float* Ms = As + KC * LDS;
        const bool low_cols = kc < 64;   // X^T[k][j] = 0 for j < k: columns 0..63 see K < 64 only
#pragma unroll 4
        for (int k = 0; k < KC; ++k) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(&As[k * LDS + 4 * ty]);
            const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(&As[k * LDS + ROWS / 2 + 4 * ty]);
            const float4 b1 = *reinterpret_cast<const float4*>(&Ms[k * LDM + 64 + 4 * tx]);
            const float bh[4] = {b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const f32x2 bb = pack2(bh[j], bh[j]);
                acc2[0][0][4 + j] = fma2(a0.x, bb, acc2[0][0][4 + j]);
                acc2[0][1][4 + j] = fma2(a0.y, bb, acc2[0][1][4 + j]);
                acc2[1][0][4 + j] = fma2(a1.x, bb, acc2[1][0][4 + j]);
                acc2[1][1][4 + j] = fma2(a1.y, bb, acc2[1][1][4 + j]);
            }
            if (low_cols) {
                const float4 b0 = *reinterpret_cast<const float4*>(&Ms[k * LDM + 4 * tx]);
                const float bl[4] = {b0.x, b0.y, b0.z, b0.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const f32x2 bb = pack2(bl[j], bl[j]);
                    acc2[0][0][j] = fma2(a0.x, bb, acc2[0][0][j]);
                    acc2[0][1][j] = fma2(a0.y, bb, acc2[0][1][j]);
                    acc2[1][0][j] = fma2(a1.x, bb, acc2[1][0][j]);
                    acc2[1][1][j] = fma2(a1.y, bb, acc2[1][1][j]);
                }
            }
        }
        __syncthreads();   // this stage is refilled
    }
    float acc[8][8];   // [row][column]
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            unpack2(acc2[i][0][j], acc[4 * i][j], acc[4 * i + 1][j]);
            unpack2(acc2[i][1][j], acc[4 * i + 2][j], acc[4 * i + 3][j]);
        }
    // epilogue: L21 = W21 D^{-1} to the factor (column-major), W21 and L21 to the staging rows (K-major)
    const float* dinv = diag_slot_d(minv, tk) + kDiagMax;
    // column col of the tile at shared column (col % 4) * 32 + col / 4: a warp's 16-byte stores fall on distinct banks
#pragma unroll
    for (int jg = 0; jg < 2; ++jg)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = 64 * jg + 4 * tx + j;
            const float di = dinv[col];
#pragma unroll
            for (int ig = 0; ig < 2; ++ig)
                *reinterpret_cast<float4*>(&psm[(j * 32 + 16 * jg + tx) * LDS + (ROWS / 2) * ig + 4 * ty]) =
                    make_float4(acc[4 * ig + 0][4 * jg + j] * di, acc[4 * ig + 1][4 * jg + j] * di,
                                acc[4 * ig + 2][4 * jg + j] * di, acc[4 * ig + 3][4 * jg + j] * di);
        }
    __syncthreads();
    {
        constexpr int LPC = ROWS / 4;   // lanes of a column
        const int lane = tid % LPC;
#pragma unroll 4
        for (int col = tid / LPC; col < nb; col += NT / LPC) {
            const float* src = &psm[((col & 3) * 32 + (col >> 2)) * LDS];
            float* dst = A + (long long)col * d.ldp;
            if (aligned && 4 * lane + 4 <= rows) {
                *reinterpret_cast<float4*>(dst + 4 * lane) = *reinterpret_cast<const float4*>(src + 4 * lane);
            } else if (aligned) {
                for (int r = 4 * lane; r < rows; ++r) dst[r] = src[r];
            } else {
                for (int r = lane; r < rows; r += LPC) dst[r] = src[r];
            }
        }
    }
    if (!tk.stage) return;
    const StageInfo g = stage_info[tk.s];
#pragma unroll
    for (int ig = 0; ig < 2; ++ig) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (ROWS / 2) * ig + 4 * ty + i;
            if (r >= rows) continue;
            const long long so = g.off + (long long)(row0 + r) * g.ld + k0;
#pragma unroll
            for (int jg = 0; jg < 2; ++jg) {
                const int col = 64 * jg + 4 * tx;
                const float* w = &acc[4 * ig + i][4 * jg];
                if (col + 4 <= nb) {
                    store_op4(stage_a + so + col, w[0], w[1], w[2], w[3]);
                    store_op4(stage_b + so + col, w[0] * dinv[col], w[1] * dinv[col + 1], w[2] * dinv[col + 2],
                              w[3] * dinv[col + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (col + j < nb) {
                            store_op1(stage_a + so + col + j, w[j]);
                            store_op1(stage_b + so + col + j, w[j] * dinv[col + j]);
                        }
                }
            }
        }
    }
    if (tk.stage_zero_to > k0 + nb) {
        const int zc = tk.stage_zero_to - (k0 + nb);
        for (int idx = tid; idx < rows * zc; idx += NT) {
            const int r = idx / zc, c = idx - r * zc;
            const long long o = g.off + (long long)(row0 + r) * g.ld + k0 + nb + c;
            store_op1(stage_a + o, 0.f);
            store_op1(stage_b + o, 0.f);
        }
    }
}

template <class F>
inline void panel_for_each(F f) {   // f(kernel, shared memory) for every instantiation
    f(k_panel_solve<float, 128>, panel_smem_bytes<128>());
    f(k_panel_solve<float, 64>, panel_smem_bytes<64>());
    f(k_panel_solve<__nv_bfloat16, 128>, panel_smem_bytes<128>());
    f(k_panel_solve<__nv_bfloat16, 64>, panel_smem_bytes<64>());
}

template <class Op>
inline void launch_panel_solve(int rows, const PanelTask* tasks, int count, const SnDev* sn, float* panel, float* minv,
                               const float* linv, Op* stage_a, Op* stage_b, const StageInfo* info, cudaStream_t st) {
    if (rows == 64)
        k_panel_solve<Op, 64><<<count, 128, panel_smem_bytes<64>(), st>>>(tasks, sn, panel, minv, linv, stage_a, stage_b, info);
    else
        k_panel_solve<Op, 128><<<count, 256, panel_smem_bytes<128>(), st>>>(tasks, sn, panel, minv, linv, stage_a, stage_b, info);
}

}  // namespace uchol_dev
