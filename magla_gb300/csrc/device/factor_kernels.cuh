// Factorisation kernels: assembly, extend-add and small fronts for both
// paths (front storage type T is double on the FP64 path, float on the mixed
// path; their pivots are FP64), and the FP64 path's pivot block, TRSM and
// right-looking updates.  The mixed path's panel kernels are in
// panel_kernels.cuh.
#pragma once

#include <cfloat>
#include <climits>
#include <cuda_bf16.h>

#include "common.cuh"
#include "plan.hpp"

namespace uchol_dev {

__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(fabs(x));
}

// max |A_ii| over the stored diagonal (ComputeDiagonalScale,
// CAESolvers/UCHOL/UtduNumericFactorization.cs:411-418).
__global__ void k_diag_scale(const double* __restrict__ values, const int* __restrict__ diag_index, int n,
                             PivotStats* st) {
    unsigned long long best = 0;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        int di = diag_index[j];
        if (di >= 0) {
            unsigned long long b = abs_bits(values[di]);
            if (b > best) best = b;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
        if (v > best) best = v;
    }
    if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(&st->min_bits, best);  // temporarily holds the scale bits
}

// Resets the statistics and turns the scale bits into the pivot controls.
__global__ void k_finish_scale(PivotStats* st, FactorCtl* ctl, double pivot_tolerance, double diagonal_regularization,
                               int allow) {
    double scale = __longlong_as_double((long long)st->min_bits);
    if (!(scale > 0.0)) scale = 1.0;
    st->scale = scale;
    st->regularized = 0;
    st->negative = 0;
    st->failed = INT_MAX;
    st->min_bits = 0x7fefffffffffffffull;  // DBL_MAX
    st->max_bits = 0;
    ctl->threshold = pivot_tolerance * scale;
    ctl->regularization = diagonal_regularization * scale;
    ctl->allow_regularization = allow;
}

// 1 / p for p > 0 without a division's FP64 instructions (64 cycles each): the FP32 reciprocal of p's leading bits as
// x0, then one third-order Newton step, x = x0 + x0 (e + e^2) with e = 1 - p x0.  |e| < 2^-22 (2^-23 for the FP32
// reciprocal's ulp, 2^-23 for the bits of p that it does not see), so the step leaves |e|^3 < 2^-66 and the roundings of e and
// e + e^2 (each below 2^-74): less than 2^-12 ulp before x is rounded, 0.5003 ulp in all.  p outside 2^+-120 is divided.
__device__ __forceinline__ double reciprocal(double p) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(p);
    const unsigned e = (unsigned)(b >> 52);
    if (e - (1023u - 120u) > 240u) return 1.0 / p;
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(((e - 1023u + 127u) << 23) | ((unsigned)(b >> 29) & 0x7fffffu))));
    const unsigned rb = __float_as_uint(r);
    const double x0 = __longlong_as_double((long long)(((unsigned long long)((rb >> 23) + (1023u - 127u)) << 52) |
                                                       ((unsigned long long)(rb & 0x7fffffu) << 29)));
    const double err = fma(-p, x0, 1.0);
    return fma(x0, fma(err, err, err), x0);
}

// Pivot acceptance exactly as the reference: !(d > tol*scale) (which also
// catches NaN) is regularised or rejected (UtduNumericFactorization.cs:557-575).
// The comparison is on the bits, which order like the numbers here: the threshold is
// not negative, a negative d has the sign bit, a NaN lies past infinity.
struct PivotAcc {
    int regularized = 0, negative = 0, failed = INT_MAX;
    unsigned long long min_bits = 0x7fefffffffffffffull, max_bits = 0;
    static __device__ __forceinline__ bool above(double piv, double threshold) {
        constexpr long long kInf = 0x7ff0000000000000ll;
        const long long t = __double_as_longlong(threshold), b = __double_as_longlong(piv);
        return b > t && b <= kInf && (unsigned long long)t <= (unsigned long long)kInf;   // a NaN threshold rejects
    }
    __device__ __forceinline__ double accept(double piv, int column, const FactorCtl& ctl) {
        if (!above(piv, ctl.threshold)) {
            if (!ctl.allow_regularization) failed = min(failed, column);
            if (piv < 0.0) ++negative;
            ++regularized;
            piv = ctl.regularization;
        }
        unsigned long long b = abs_bits(piv);
        if (b < min_bits) min_bits = b;
        if (b > max_bits) max_bits = b;
        return piv;
    }
    __device__ __forceinline__ void flush(PivotStats* st) const {
        if (regularized) atomicAdd(&st->regularized, regularized);
        if (negative) atomicAdd(&st->negative, negative);
        if (failed != INT_MAX) atomicMin(&st->failed, failed);
        atomicMin(&st->min_bits, min_bits);
        atomicMax(&st->max_bits, max_bits);
    }
};

template <class T>
__global__ void k_assemble(const double* __restrict__ values, const long long* __restrict__ pos, int nnz,
                           T* __restrict__ panel) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x)
        panel[pos[k]] = (T)values[k];
}

// Extend-add: one warp per receiving parent column; the children's columns
// that land in it are added in child order (deterministic, no atomics).
// UtduNumericFactorization.cs:471-509.  A column of the parent's contribution
// block starts from zero (the reference zeroes the whole front, :441-447; only
// the lower triangle is ever read): its first child's column is written out
// together with the zeros between its entries, window by window of kEaWindow
// rows through shared memory, so that every row is written once.  (Clearing the
// column first and adding to it afterwards let 6,000 warps' columns leave L2 in
// between: the traffic of a 10,000-row front was twice the bytes.)  Later
// children, and columns of the panel, which hold the assembled values, are
// added to what is there.  HBM bounds it.
// Side = true: the instance launched on the side stream (its graph nodes run at
// the lowest priority, so that the main stream's CTAs are scheduled first).
constexpr int kEaWindow = 256, kEaThreads = 256;
template <class T, bool Side = false>
__global__ void __launch_bounds__(kEaThreads) k_extend_add(const EaItem* __restrict__ items, int count,
                                                           const EaEntry* __restrict__ entries, const SnDev* __restrict__ sn,
                                                           const int* __restrict__ rel, T* __restrict__ panel,
                                                           T* __restrict__ contrib) {
    __shared__ __align__(16) T windows[kEaThreads / 32][kEaWindow];
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (kEaThreads >> 5);
    constexpr int D = kEaWindow / 32;   // loads of a batch in flight per lane
    for (int warp = (blockIdx.x * kEaThreads + threadIdx.x) >> 5; warp < count; warp += warps) {
        const EaItem it = items[warp];
        const SnDev P = sn[it.parent];
        T* dst;
        int shift, first = it.begin;
        if (it.pcol < P.w) {
            dst = panel + P.panel_off + (long long)it.pcol * P.ldp;
            shift = 0;
        } else {
            const int c = it.pcol - P.w, t = P.m - P.w;
            dst = contrib + P.contrib_off + (long long)c * P.ldc;
            shift = P.w;
            T* win = windows[threadIdx.x >> 5];
            const int* r = rel;
            const T* src = nullptr;
            int b = 0, bt = 0;   // the first child's entries still to come
            if (first < it.end) {
                const EaEntry en = entries[first++];
                const SnDev C = sn[en.child];
                r += C.rel_off;
                src = contrib + C.contrib_off + (long long)en.a * C.ldc;
                b = en.a;
                bt = C.m - C.w;
            }
            // rows [c, t) in windows that start on multiples of kEaWindow (the column starts on a 16-byte boundary:
            // contribution offsets are multiples of 64 elements, ldc of 8)
            for (int R = c / kEaWindow * kEaWindow; R < t; R += kEaWindow) {
                constexpr int V = 16 / (int)sizeof(T);
                for (int v = lane; v < kEaWindow / V; v += 32) reinterpret_cast<uint4*>(win)[v] = make_uint4(0u, 0u, 0u, 0u);
                __syncwarp();
                int taken = 0;
                if (b < bt) {
                    int idx[D];
                    T sv[D];
#pragma unroll
                    for (int u = 0; u < D; ++u) {
                        const int q = b + lane + 32 * u;
                        idx[u] = q < bt ? r[q] - shift - R : kEaWindow;   // ascending, so at most kEaWindow of them here
                        sv[u] = q < bt ? src[q] : T(0);
                    }
#pragma unroll
                    for (int u = 0; u < D; ++u) {
                        const bool in = idx[u] < kEaWindow;
                        if (in) win[idx[u]] = sv[u];
                        taken += __popc(__ballot_sync(0xffffffffu, in));
                    }
                    __syncwarp();
                }
                b += taken;
                const int lo = max(c, R), hi = min(t, R + kEaWindow);
                for (int v = R / V + lane; v < (R + kEaWindow) / V; v += 32) {
                    const int e = v * V;
                    if (e >= lo && e + V <= hi) {
                        reinterpret_cast<uint4*>(dst)[v] = reinterpret_cast<const uint4*>(win)[v - R / V];
                    } else {
#pragma unroll
                        for (int k = 0; k < V; ++k)
                            if (e + k >= lo && e + k < hi) dst[e + k] = win[e + k - R];
                    }
                }
                __syncwarp();
            }
        }
        for (int e = first; e < it.end; ++e) {
            const EaEntry en = entries[e];
            const SnDev C = sn[en.child];
            const int t = C.m - C.w;
            const int* r = rel + C.rel_off;
            const T* src = contrib + C.contrib_off + (long long)en.a * C.ldc;
            // rows of one child column are distinct, so loads of a batch are issued before its stores
            for (int b0 = en.a + lane; b0 < t; b0 += 32 * D) {
                int idx[D];
                T sv[D], dv[D];
#pragma unroll
                for (int u = 0; u < D; ++u) {
                    const int b = b0 + 32 * u;
                    idx[u] = b < t ? r[b] - shift : -1;
                    sv[u] = b < t ? src[b] : T(0);
                }
#pragma unroll
                for (int u = 0; u < D; ++u) dv[u] = idx[u] >= 0 ? dst[idx[u]] : T(0);
#pragma unroll
                for (int u = 0; u < D; ++u)
                    if (idx[u] >= 0) dst[idx[u]] = dv[u] + sv[u];
            }
            __syncwarp();
        }
    }
}

// ---- FP64 pivots, panels and updates ----
//
// What bounds them: the FP64 pipe.  A scheduler issues one FP64 warp instruction per 64 cycles, however few of its
// lanes are active, so an SM does two multiply-adds per clock: a 64 x 64 x 32 update tile alone takes one SM 32 us,
// a 128-row panel solve 16 us, a division about ten instructions.  So work is cut fine enough to reach every SM
// (16- and 32-row tiles), operands take one multiply-add per entry (the unscaled column times L, no separate
// product with the pivot), and the chain of pivots has a warp, and as far as possible a scheduler, to itself.

// Small fronts (m <= LW): LW lanes a front, lane = row, the front's rows in registers.  The row is a shift register
// (a[j] is column k + j at pivot k), so every register index is a constant while the pivots' loop stays rolled.
constexpr int kLaneFrontThreads = 128;
template <class T, int LW>
__global__ void __launch_bounds__(kLaneFrontThreads) k_small_fronts_lanes(const int* __restrict__ fronts, int count,
                                                                         const SnDev* __restrict__ sn, T* __restrict__ panel,
                                                                         T* __restrict__ contrib, double* __restrict__ diag,
                                                                         const FactorCtl* __restrict__ ctlp, PivotStats* st) {
    const int r = threadIdx.x & (LW - 1), q = (blockIdx.x * kLaneFrontThreads + threadIdx.x) / LW;
    const FactorCtl ctl = *ctlp;
    SnDev d{};   // m = w = 0 past the last front
    if (q < count) d = sn[fronts[q]];
    const int m = d.m, w = d.w;
    T* P = panel + d.panel_off;
    T* C = contrib + d.contrib_off;
    double a[LW];
#pragma unroll
    for (int j = 0; j < LW; ++j)
        a[j] = r < m && j <= r ? (j < w ? (double)P[r + (long long)j * d.ldp] : (double)C[(r - w) + (long long)(j - w) * d.ldc]) : 0.0;
    int wmax = w, mmax = m;
    for (int o = 16; o >= LW && o > 0; o >>= 1) {
        wmax = max(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
        mmax = max(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
    }
    PivotAcc acc;
    for (int k = 0; k < wmax; ++k) {
        const bool live = k < w;   // the same in the front's lanes
        const double raw = __shfl_sync(0xffffffffu, a[0], k, LW);
        const double piv = live ? acc.accept(raw, d.first_col + k, ctl) : 1.0;
        const double inv = reciprocal(piv);
        const double wk = a[0];
        const double l = live && r > k && r < m ? wk * inv : 0.0;
        if (live && r >= k && r < m) P[r + (long long)k * d.ldp] = r == k ? (T)1 : (T)l;
        if (live && r == k) diag[d.first_col + k] = piv;
        const int rem = mmax - 1 - k;
#pragma unroll
        for (int j = 1; j < LW; ++j) {
            if (j > rem) break;
            const double wj = __shfl_sync(0xffffffffu, wk, (k + j) & (LW - 1), LW);
            const double v = fma(-l, wj, a[j]);
            if (live) a[j - 1] = v;
        }
    }
#pragma unroll
    for (int j = 0; j < LW; ++j)   // column w + j of the contribution
        if (w + j <= r && r < m) C[(r - w) + (long long)j * d.ldc] = (T)a[j];
    // statistics: one set of atomics a warp
    if (r != 0) acc = PivotAcc();
    for (int o = 16; o > 0; o >>= 1) {
        acc.regularized += __shfl_xor_sync(0xffffffffu, acc.regularized, o);
        acc.negative += __shfl_xor_sync(0xffffffffu, acc.negative, o);
        acc.failed = min(acc.failed, __shfl_xor_sync(0xffffffffu, acc.failed, o));
        acc.min_bits = min(acc.min_bits, __shfl_xor_sync(0xffffffffu, acc.min_bits, o));
        acc.max_bits = max(acc.max_bits, __shfl_xor_sync(0xffffffffu, acc.max_bits, o));
    }
    if ((threadIdx.x & 31) == 0) acc.flush(st);
}

// LDL^T of the first w columns of the m x m matrix at S (column-major, leading dimension ld, lower triangle,
// m <= 32 NQ) in shared memory, by kWarps warps: warp 0 is the chain (its current column in registers: pivot,
// reciprocal, the scaled column, the next column's update), the others update the columns after that, four at a time
// (loads of all four, then the products, then the stores: one at a time, the latencies of one column after another
// made the others the chain's bottleneck); one barrier a pivot.  Wc: two buffers of wstride entries for the unscaled
// column.
template <int kWarps, int NQ, class Pivot>
__device__ __forceinline__ void smem_ldlt(double* S, int ld, int m, int w, double* Wc, int wstride, Pivot&& pivot) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        double c[NQ];   // rows lane + 32 q of the current column
#pragma unroll
        for (int q = 0; q < NQ; ++q) c[q] = lane + 32 * q < m ? S[lane + 32 * q] : 0.0;
        for (int k = 0; k < w; ++k) {
            double* W = Wc + (k & 1) * wstride;
            double* Lk = S + (long long)k * ld;
            double mine = 0.0, after = 0.0;   // rows k and k + 1 of the column, in their lanes
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (q == k >> 5) mine = c[q];
                if (q == (k + 1) >> 5) after = c[q];
            }
            const double piv = pivot(k, __shfl_sync(0xffffffffu, mine, k & 31));
            const double wj = __shfl_sync(0xffffffffu, after, (k + 1) & 31);
            const double inv = reciprocal(piv);
            double l[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int i = lane + 32 * q;
                if (32 * q + 31 <= k || 32 * q >= m) continue;
                l[q] = i == k ? 1.0 : c[q] * inv;
                if (i >= k && i < m) {
                    W[i] = c[q];
                    Lk[i] = l[q];
                }
            }
            if (k % 32 == 31 && lane == 31) Lk[k] = 1.0;   // row k is the last of a group that the loop left out
            __syncthreads();
            if (k + 1 < w) {
                const double* n = S + (long long)(k + 1) * ld;
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const int i = lane + 32 * q;
                    if (32 * q + 31 <= k || 32 * q >= m) continue;
                    c[q] = fma(-l[q], wj, i < m ? n[i] : 0.0);
                }
            }
        }
    } else {
        for (int k = 0; k < w; ++k) {
            __syncthreads();
            const double* W = Wc + (k & 1) * wstride;
            const double* Lk = S + (long long)k * ld;
            const int first = k + 1 + (k + 1 < w ? 1 : 0) + warp - 1;   // the next column is the chain's
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int i = lane + 32 * q, last = min(m - 1, 32 * q + 31);   // columns up to this group's last row
                if (32 * q >= m || first > last) continue;
                const double li = i > k && i < m ? Lk[i] : 0.0;
                for (int j = first; j <= last; j += 4 * (kWarps - 1)) {
                    double v[4], x[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int jj = j + u * (kWarps - 1);
                        const bool on = jj <= last;
                        x[u] = on ? W[jj] : 0.0;
                        v[u] = on && i >= jj && i < m ? S[i + (long long)jj * ld] : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int jj = j + u * (kWarps - 1);
                        if (jj > last) break;
                        v[u] = fma(-li, x[u], v[u]);
                        if (i >= jj && i < m) S[i + (long long)jj * ld] = v[u];
                    }
                }
            }
        }
    }
    __syncthreads();
}

// Whole front of 32 < m <= kSmallFrontLimit rows in shared memory (FP64); writes the unit factor block and the
// contribution.
constexpr int kSmallFrontThreads = 256;
__host__ __device__ constexpr size_t small_front_smem(int m) { return ((size_t)m * m + 2 * (size_t)m) * sizeof(double); }
template <class T>
__global__ void __launch_bounds__(kSmallFrontThreads) k_small_fronts(const int* __restrict__ fronts, const SnDev* __restrict__ sn,
                                                                     T* __restrict__ panel, T* __restrict__ contrib,
                                                                     double* __restrict__ diag, const FactorCtl* __restrict__ ctlp,
                                                                     PivotStats* st) {
    extern __shared__ double S[];
    const SnDev d = sn[fronts[blockIdx.x]];
    const FactorCtl ctl = *ctlp;
    const int m = d.m, w = d.w, ld = m;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kSmallFrontThreads / 32;
    T* P = panel + d.panel_off;
    T* C = contrib + d.contrib_off;
    for (int j = warp; j < m; j += kWarps) {
        const T* src = j < w ? P + (long long)j * d.ldp : C + (long long)(j - w) * d.ldc - w;
#pragma unroll 4
        for (int i = j + lane; i < m; i += 32) S[i + j * ld] = (double)src[i];
    }
    PivotAcc acc;
    __syncthreads();
    smem_ldlt<kWarps, kSmallFrontLimit / 32>(S, ld, m, w, S + (size_t)m * m, m, [&](int k, double raw) {
        const double piv = acc.accept(raw, d.first_col + k, ctl);
        if (lane == 0) diag[d.first_col + k] = piv;
        return piv;
    });
    for (int j = warp; j < m; j += kWarps) {
        T* dst = j < w ? P + (long long)j * d.ldp : C + (long long)(j - w) * d.ldc - w;
#pragma unroll 4
        for (int i = j + lane; i < m; i += 32) dst[i] = (T)S[i + j * ld];
    }
    if (threadIdx.x == 0) acc.flush(st);
}

// Pivot block [j0, j0+nb) of a large front: FP64 LDL^T of the nb x nb
// diagonal block in shared memory, one CTA per block; writes the unit L11,
// the pivots D and the statistics (UtduNumericFactorization.cs:553-592
// restricted to the diagonal block).
constexpr int kMaxPivotBlock = 64, kPivotThreads = 256;

template <class T>
__global__ void __launch_bounds__(kPivotThreads) k_pivot_block(const PanelTask* __restrict__ tasks, const SnDev* __restrict__ sn,
                                                     T* __restrict__ panel, double* __restrict__ diag,
                                                     const FactorCtl* __restrict__ ctlp, PivotStats* st) {
    __shared__ double Dg[kMaxPivotBlock * (kMaxPivotBlock + 1)];
    __shared__ double Wc[2 * kMaxPivotBlock];
    const PanelTask tk = tasks[blockIdx.x];
    const SnDev d = sn[tk.s];
    const FactorCtl ctl = *ctlp;
    const int nb = tk.nb, j0 = tk.j0, ld = kMaxPivotBlock + 1;
    const int tid = threadIdx.x, lane = tid & 31;
    T* P = panel + d.panel_off + j0 + (long long)j0 * d.ldp;
#pragma unroll 4
    for (int e = tid; e < kMaxPivotBlock * nb; e += kPivotThreads) {
        const int r = e % kMaxPivotBlock, c = e / kMaxPivotBlock;
        if (r >= c && r < nb) Dg[r + c * ld] = (double)P[r + (long long)c * d.ldp];
    }
    PivotAcc acc;
    __syncthreads();
    smem_ldlt<kPivotThreads / 32, kMaxPivotBlock / 32>(Dg, ld, nb, nb, Wc, kMaxPivotBlock, [&](int k, double raw) {
        const double piv = acc.accept(raw, d.first_col + j0 + k, ctl);
        if (lane == 0) diag[d.first_col + j0 + k] = piv;
        return piv;
    });
#pragma unroll 4
    for (int e = tid; e < kMaxPivotBlock * nb; e += kPivotThreads) {
        const int r = e % kMaxPivotBlock, c = e / kMaxPivotBlock;
        if (r >= c && r < nb) P[r + (long long)c * d.ldp] = (T)Dg[r + c * ld];
    }
    if (tid == 0) acc.flush(st);
}

// Rows under the pivot block (FP64 path): Y = F21 L11^-T (forward substitution
// per row), L21 = Y / D.  Eight lanes a row, lane q holding columns q, q + 8, ...
// (at pivot column k each lane has at most NBMAX / 8 - k / 8 entries to update:
// 80 multiply-adds a lane for 32 columns where a thread per row takes 496 one
// after another, 16 us); kTrsmRows rows a CTA, kTrsmSplit CTAs a task.
constexpr int kTrsmRows = 16, kTrsmSplit = 128 / kTrsmRows;
template <class T, int NBMAX>
__global__ void __launch_bounds__(128) k_trsm(const PanelTask* __restrict__ tasks, const SnDev* __restrict__ sn,
                                              T* __restrict__ panel, const double* __restrict__ diag) {
    constexpr int NC = NBMAX / 8;
    __shared__ double L11[NBMAX * (NBMAX + 1)];   // L11[k * (NBMAX + 1) + c], zero for c <= k
    __shared__ double dinv[NBMAX];
    const PanelTask tk = tasks[blockIdx.x / kTrsmSplit];
    const int sub = blockIdx.x % kTrsmSplit * kTrsmRows;
    if (sub >= tk.rows) return;
    const SnDev d = sn[tk.s];
    const int nb = tk.nb, j0 = tk.j0, ld = NBMAX + 1;
    const int tid = threadIdx.x, lane = tid & 31, q = lane >> 2;
    const int row = sub + 4 * (tid >> 5) + (lane & 3), i = tk.row0 + row;
    T* P = panel + d.panel_off + (long long)j0 * d.ldp;
    const bool live = row < tk.rows;
    double a[NC];
#pragma unroll
    for (int t = 0; t < NC; ++t) a[t] = live && q + 8 * t < nb ? (double)P[i + (long long)(q + 8 * t) * d.ldp] : 0.0;
#pragma unroll 8
    for (int e = tid; e < NBMAX * NBMAX; e += 128) {
        const int r = e % NBMAX, c = e / NBMAX;   // L(r, c)
        L11[c * ld + r] = r > c && r < nb ? (double)P[j0 + r + (long long)c * d.ldp] : 0.0;
    }
    if (tid < NBMAX) dinv[tid] = tid < nb ? reciprocal(diag[d.first_col + j0 + tid]) : 0.0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NBMAX; ++k) {
        if (k >= nb) break;
        const double y = __shfl_sync(0xffffffffu, a[k / 8], (lane & 3) + 4 * (k & 7));
#pragma unroll
        for (int t = k / 8; t < NC; ++t) a[t] = fma(-y, L11[k * ld + q + 8 * t], a[t]);
    }
#pragma unroll
    for (int t = 0; t < NC; ++t)
        if (live && q + 8 * t < nb) P[i + (long long)(q + 8 * t) * d.ldp] = (T)(a[t] * dinv[q + 8 * t]);
}

// Update C[i, j] -= sum_k L[i,k] d_k L[j,k] of one TS x TS tile (lower triangle, i >= j), TS = 16 or 32: 2 or 8 us of
// the SM's FP64 pipe at 32 columns (Launch::variant: 32 once that still makes two CTAs per SM).  Consecutive threads
// hold consecutive rows of C.
template <int TS>
__host__ __device__ constexpr int simt_threads() { return 128; }   // a warp per scheduler
template <class T, int TS>
__global__ void __launch_bounds__(simt_threads<TS>()) k_simt_update(const UpdJob* __restrict__ jobs, int njobs,
                                                                   const SnDev* __restrict__ sn, T* __restrict__ panel,
                                                                   T* __restrict__ contrib, const double* __restrict__ diag) {
    constexpr int KC = 32, NT = simt_threads<TS>(), NY = NT / 16, PI = TS / 16, QJ = TS / NY;   // rows, columns of a thread
    __shared__ double As[KC][TS];
    __shared__ double Bs[KC][TS];
    const UpdJob J = jobs[find_job(jobs, njobs, blockIdx.x)];
    const SnDev d = sn[J.s];
    int i0, j0, jend;
    decode_tile(J, d, TS, (long long)blockIdx.x - J.tile_begin, i0, j0, jend);
    const T* Pn = panel + d.panel_off;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // the tile's entries of C, in flight during the products
    const bool in_panel = j0 < d.w;
    T* base = in_panel ? panel : contrib;
    long long off[PI][QJ];
    double old[PI][QJ], acc[PI][QJ];
#pragma unroll
    for (int q = 0; q < QJ; ++q)
#pragma unroll
        for (int p = 0; p < PI; ++p) {
            const int j = j0 + ty + NY * q, i = i0 + tx + 16 * p;
            const bool ok = j < jend && i < d.m && i >= j;
            off[p][q] = !ok ? -1
                            : in_panel ? d.panel_off + i + (long long)j * d.ldp
                                       : d.contrib_off + (i - d.w) + (long long)(j - d.w) * d.ldc;
            old[p][q] = ok ? (double)base[off[p][q]] : 0.0;
            acc[p][q] = 0.0;
        }
    for (int kc = 0; kc < J.kn; kc += KC) {
        const int kl = min(KC, J.kn - kc);
        if (kc > 0) __syncthreads();
#pragma unroll 4
        for (int idx = threadIdx.x; idx < KC * TS; idx += NT) {
            const int r = idx % TS, k = idx / TS, kk = J.k0 + kc + k;
            double av = 0.0, bv = 0.0;
            if (k < kl) {
                const int i = i0 + r, j = j0 + r;
                if (i < d.m) av = (double)Pn[i + (long long)kk * d.ldp];
                if (j < d.m) bv = (double)Pn[j + (long long)kk * d.ldp] * diag[d.first_col + kk];
            }
            As[k][r] = av;
            Bs[k][r] = bv;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < kl; ++k) {
            double a[PI], b[QJ];
#pragma unroll
            for (int p = 0; p < PI; ++p) a[p] = As[k][tx + 16 * p];
#pragma unroll
            for (int q = 0; q < QJ; ++q) b[q] = Bs[k][ty + NY * q];
#pragma unroll
            for (int p = 0; p < PI; ++p)
#pragma unroll
                for (int q = 0; q < QJ; ++q) acc[p][q] = fma(a[p], b[q], acc[p][q]);
        }
    }
#pragma unroll
    for (int q = 0; q < QJ; ++q)
#pragma unroll
        for (int p = 0; p < PI; ++p)
            if (off[p][q] >= 0) base[off[p][q]] = (T)(old[p][q] - acc[p][q]);
}

}  // namespace uchol_dev
