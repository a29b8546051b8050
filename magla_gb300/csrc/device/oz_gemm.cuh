// FP64 Schur update on the tensor cores: C -= L W^T (W = L D, rounded to FP64) over a front's trailing lower triangle,
// with every FP64 entry of L and W split into eight 8-bit digits that the BF16 tensor cores multiply without error (the
// scheme of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix multiplication", 2012, on fixed-point
// slices).
//
// Why: the FP64 pipe does two multiply-adds a clock and SM (1.25 TFLOP/s on the GPU); the update is a contraction, and
// 36 exact digit products at 1.9 PFLOP/s are worth 40 times that.  What bounds it: an SM's shared-memory path (a
// 128 x 64 tile reads 6 KB per 16-deep product) and the accumulators' read-out.  30^3 elasticity, 5.4e11 operations:
// 500 ms on the FP64 pipe (1.07 TFLOP/s), 32.6 ms here.
//
// Slices.  Column k of L is scaled by 2^s and of W by 2^-s, s about log2(d_k) / 2 (exact; both are then of the size of
// L sqrt(D), so that no column of the chunk is small in one and large in the other).  For each row i of either and chunk
// of 128 columns (K), E_i is the largest exponent of the row's scaled entries and X = round(a 2^(63 - E_i)) a 64-bit
// integer (|a| < 2^E_i), written in balanced base 256: X = sum_p d_p 2^(8 (7 - p)), |d_p| <= 128.  The product of two rows
// over a chunk is 2^(E_i + E_j - 126) sum_{p, q} 2^(8 (14 - p - q)) d_p . d_q; the orders o = p + q <= 7 are kept.  One
// FP32 accumulator per order: at most 8 products of 128 terms of at most 2^14 each, so every partial sum is an integer of
// at most 2^24 and exact.  The eight sums are joined in a 64-bit integer whose unit follows the size of the result
// (2^-60 of it), rounded to FP64 and added to the tile's FP64 sums, chunk by chunk; C takes one FP64 subtraction.
// Every tile is one CTA's: the result is deterministic.
//
// What is lost.  The orders past 7 are 2^-60.7 2^(E_i + E_j) in the mean of random digits and below 2^-54 2^(E_i + E_j)
// whatever the digits; an entry 2^-11 of its row's largest or smaller starts to lose low bits of its own.  FP64 sums lose
// 2^-53 of sum_k |l_ik d_k l_jk|, so the digits are the more accurate where that sum is above 2^-7 of the product of the
// rows' largest entries, and the less accurate entry by entry where two rows have their large entries in different
// columns.  Against sqrt(c_ii c_jj), which is at least that product and in which the error of a Cholesky factorisation
// is measured (the same under every scaling of the equations), every entry's loss is below FP64's unit roundoff.
//
// Layout: staging rows (front rows) of 512 bytes per 32 columns: eight slices of 32 BF16 digits, so that a 128-byte
// swizzled box holds two slices of 32 columns.
#pragma once

#include "tc_gemm.cuh"

namespace uchol_dev {

constexpr int kOzCols = 64, kOzRows = 2 * kOzCols;   // tile of C: columns x rows
constexpr int kOzChunk = 128;        // columns (K) that share a row's exponent and an accumulator round
constexpr int kOzGroup = 32;         // columns per staging group (one ring stage)
constexpr int kOzSlices = 8;
constexpr int kOzGroupElems = kOzSlices * kOzGroup;
constexpr int kOzStages = 2;
constexpr int kOzABytes = kOzSlices / 2 * kOzRows * 128, kOzBBytes = kOzSlices / 2 * kOzCols * 128;
constexpr int kOzThreads = 64 + 256;   // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int kOzNan = 1 << 20;      // row exponent of a chunk with an entry that is not finite
constexpr int kOzZeroRow = 1023;     // and of one without digits (any value)
// Two row exponents from kOzLow to kOzHigh put every nonzero integer of the epilogue into the range of normal doubles.
constexpr int kOzLow = 600, kOzHigh = 1500;

inline size_t oz_smem_bytes() { return 1024 + (size_t)kOzStages * (kOzABytes + kOzBBytes) + 128; }

// 8 accumulator columns of this thread's TMEM lane (no wait).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Digits of columns [j0, j0 + nb) (one chunk) of the panel rows [row0, row0 + rows) of a front into its staging rows of
// L and W, and the rows' exponents (those of W after all of L's); 32 rows a CTA, kOzSplit CTAs a task.
constexpr int kOzSliceRows = 32, kOzSplit = 128 / kOzSliceRows;
__global__ void __launch_bounds__(256) k_oz_slice(const PanelTask* __restrict__ tasks, const SnDev* __restrict__ sn,
                                                  const double* __restrict__ panel, const double* __restrict__ diag,
                                                  __nv_bfloat16* __restrict__ stage_l, __nv_bfloat16* __restrict__ stage_w,
                                                  int* __restrict__ exps, long long w_exps,
                                                  const StageInfo* __restrict__ stage_info) {
    constexpr int LD = kOzSliceRows + 1;
    __shared__ double A[kOzChunk * LD];
    __shared__ double D[kOzChunk];
    const PanelTask tk = tasks[blockIdx.x / kOzSplit];
    const int sub = blockIdx.x % kOzSplit * kOzSliceRows;
    if (sub >= tk.rows) return;
    const SnDev d = sn[tk.s];
    const StageInfo g = stage_info[tk.s];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row0 = tk.row0 + sub, rows = min(kOzSliceRows, tk.rows - sub);
    if (tid < kOzChunk) D[tid] = tid < tk.nb ? diag[d.first_col + tk.j0 + tid] : 1.0;
    const double* P = panel + d.panel_off + row0 + (long long)tk.j0 * d.ldp;
#pragma unroll 4
    for (int k = warp; k < kOzChunk; k += 8) A[k * LD + lane] = lane < rows && k < tk.nb ? P[lane + (long long)k * d.ldp] : 0.0;
    __syncthreads();
    const int groups = (tk.nb + kOzGroup - 1) / kOzGroup;
    double dk[4];
    int scale[4];   // s of this lane's columns
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        dk[q] = D[32 * q + lane];
        scale[q] = ((int)((__double_as_longlong(dk[q]) >> 52) & 0x7ff) - 1023) >> 1;
    }
    for (int r = warp; r < rows; r += 8)
#pragma unroll
        for (int side = 0; side < 2; ++side) {   // L, W
            long long b[4];
            int e[4], E = -100000, least = 1;
            bool finite = true;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double l = A[(32 * q + lane) * LD + r];
                b[q] = __double_as_longlong(side ? l * dk[q] : l);
                const int raw = (int)((b[q] >> 52) & 0x7ff);
                finite = finite && raw != 0x7ff;
                least = min(least, raw);
                e[q] = raw + (side ? -scale[q] : scale[q]);
            }
            if (__any_sync(0xffffffffu, least == 0)) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const long long frac = b[q] & 0xfffffffffffffll;
                    if (((b[q] >> 52) & 0x7ff) != 0) continue;
                    if (frac == 0) {
                        e[q] = -100000;
                    } else {   // subnormal: its leading bit to 52
                        const int z = __clzll(frac) - 11;
                        b[q] = (b[q] & (1ll << 63)) | (frac << z);
                        e[q] += 1 - z;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) E = max(E, e[q]);
            for (int o = 16; o > 0; o >>= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
            const bool all_finite = __all_sync(0xffffffffu, finite);
            if (lane == 0)
                exps[(side ? w_exps : 0) + g.eoff + (long long)(tk.j0 / kOzChunk) * d.ldp + row0 + r] =
                    !all_finite ? kOzNan : E <= -50000 ? kOzZeroRow : E;
            __nv_bfloat16* out = (side ? stage_w : stage_l) + g.off + (long long)(row0 + r) * g.ld +
                                 (long long)(tk.j0 / kOzGroup) * kOzGroupElems + lane;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q >= groups) break;
                const int sh = e[q] - E + 10;   // X = M 2^sh, M the 53-bit significand
                const unsigned long long M = ((unsigned long long)b[q] & 0xfffffffffffffull) | 0x10000000000000ull;
                long long X = e[q] <= -50000 || sh < -54 ? 0 : (long long)(sh >= 0 ? M << sh : (M + (1ull << (-sh - 1))) >> -sh);
                if (b[q] < 0) X = -X;
#pragma unroll
                for (int p = kOzSlices - 1; p >= 0; --p) {
                    const int digit = p > 0 ? (int)(signed char)(X & 0xff) : (int)X;
                    X = (X - digit) >> 8;
                    out[q * kOzGroupElems + p * kOzGroup] = __float2bfloat16_rn((float)digit);   // at most 8 bits: exact
                }
            }
        }
}

__device__ __forceinline__ int oz_int(uint32_t r) { return __float2int_rn(__uint_as_float(r)); }   // an integer's FP32

// The value V 2^(sh) as a double (V a 64-bit integer, rounded once, and once more if the result is subnormal), zero or
// infinite past the range of doubles.
__device__ __forceinline__ double oz_value(long long V, int sh) {
    const long long b = __double_as_longlong((double)V);
    const int e = (int)((b >> 52) & 0x7ff) + sh;
    if (V == 0 || e < -63) return 0.0;
    if (e <= 0) return __longlong_as_double(b + ((long long)(sh + 64) << 52)) * 0x1p-64;
    return e >= 0x7ff ? __longlong_as_double((b & (1ll << 63)) | 0x7ff0000000000000ll) : __longlong_as_double(b + ((long long)sh << 52));
}

// Jobs as k_tc_gemm's, in tiles of 64 columns x 128 rows (one CTA each); maps 2 map (128-row box of the front's L rows)
// and 2 map + 1 (64-row box of its W rows).
__global__ void __launch_bounds__(kOzThreads, 1)
    k_oz_gemm(const TcJob* __restrict__ jobs, int njobs, const SnDev* __restrict__ sn, double* __restrict__ panel,
              double* __restrict__ contrib, const CUtensorMap* __restrict__ maps, const int* __restrict__ exps,
              long long w_exps, const StageInfo* __restrict__ stage_info, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + kOzStages * kOzABytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sB + kOzStages * kOzBBytes);
    uint64_t* empty = full + kOzStages;
    uint64_t* acc_full = empty + kOzStages;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int q = 0; q < kOzStages; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kOzThreads - 64);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto fail = [&]() {
        atomicExch(status, kTcStatusTimeout);
        *abort_flag = 1;
    };
    const TcJob J = jobs[tc_find_job(jobs, njobs, blockIdx.x)];
    const SnDev d = sn[J.s];
    int i0, j0, jend;
    tc_decode_tile<kOzCols>(J.c0, J.cend, d.m, (long long)blockIdx.x - J.tile_begin, i0, j0, jend);
    const int g0 = J.kbeg / kOzGroup, g1 = (J.kbeg + J.kn + kOzGroup - 1) / kOzGroup;   // staging groups of the sum
    constexpr int kPerChunk = kOzChunk / kOzGroup;

    if (warp == 0) {
        if (lane == 0) {
            const CUtensorMap* ma = maps + 2 * J.map;
            const CUtensorMap* mb = ma + 1;
            int stage = 0;
            uint32_t phase = 0;
            for (int g = g0; g < g1 && !*abort_flag; ++g) {
                if (!mbar_wait(&empty[stage], phase ^ 1)) { fail(); break; }
                mbar_arrive_expect_tx(&full[stage], kOzABytes + kOzBBytes);
#pragma unroll
                for (int p = 0; p < kOzSlices / 2; ++p) {
                    const int x = g * kOzGroupElems + p * 64;
                    tma_load_2d(sA + stage * kOzABytes + p * kOzRows * 128, ma, &full[stage], x, i0);
                    tma_load_2d(sB + stage * kOzBBytes + p * kOzCols * 128, mb, &full[stage], x, j0);
                }
                if (++stage == kOzStages) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = mma_idesc(1u, kOzRows, kOzCols);
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int c = g0; c < g1 && ok && !*abort_flag; c += kPerChunk) {
                if (!mbar_wait(acc_empty, acc_phase ^ 1)) { fail(); break; }
                tc_fence_after();
                const int ce = min(g1, c + kPerChunk);
                for (int g = c; g < ce; ++g) {
                    if (!mbar_wait(&full[stage], phase)) { fail(); ok = false; break; }
                    tc_fence_after();
                    const uint32_t a0 = smem_u32(sA + stage * kOzABytes), b0 = smem_u32(sB + stage * kOzBBytes);
#pragma unroll
                    for (int p = 0; p < kOzSlices; ++p)
#pragma unroll
                        for (int q = 0; q < kOzSlices - p; ++q)
#pragma unroll
                            for (int kk = 0; kk < 2; ++kk)
                                umma<true>(tmem + (uint32_t)((p + q) * kOzCols),
                                           sw128_desc(a0 + (p >> 1) * kOzRows * 128 + (p & 1) * 64 + kk * 32),
                                           sw128_desc(b0 + (q >> 1) * kOzCols * 128 + (q & 1) * 64 + kk * 32), idesc,
                                           (g != c || p != 0 || kk != 0) ? 1u : 0u);   // (0, q) comes first of order q
                    umma_commit(&empty[stage]);
                    if (++stage == kOzStages) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                umma_commit(acc_full);
                acc_phase ^= 1;
            }
        }
    } else {
        // epilogue: thread = row (its TMEM lane) and half of the columns
        const int quad = warp & 3, half = (warp - 2) >> 2, i = i0 + 32 * quad + lane, jb = j0 + 32 * half;
        const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(32 * half);
        const int* ex = exps + stage_info[J.s].eoff;
        double sum[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) sum[c] = 0.0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int c = g0; c < g1 && ok; c += kPerChunk) {
            const long long eo = (long long)(c / kPerChunk) * d.ldp;
            const int ei = i < d.m ? ex[eo + i] : kOzZeroRow, ejl = jb + lane < d.m ? ex[w_exps + eo + jb + lane] : kOzZeroRow;
            const bool normal = __all_sync(0xffffffffu, min(ei, ejl) >= kOzLow && max(ei, ejl) <= kOzHigh);
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full, acc_phase));
            if (!ok) {
                fail();
                break;
            }
            acc_phase ^= 1;
            tc_fence_after();
            // T = the sum over the orders, in units of order 7: its upper half hi (orders 0 to 3, units of order 3, below
            // 2^45.1) and its lower half lo (orders 4 to 7, below 2^47.4), which carries into hi.  T is held as V 2^(32 - k), V
            // its leading 64 bits: k, from 17 to 31, shifts out hi's copies of the sign.  This stands between the products
            // of one chunk and the next, so its instructions count: 64-bit shifts and a rounding here were 2 ms of the
            // 30^3 elasticity step
            long long V[32];
            unsigned ks[4] = {0u, 0u, 0u, 0u};   // k - 16 of each entry, four bits
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t r0[8], r1[8], r2[8], r3[8];
                tmem_ld8(ta + 0 * kOzCols + 8 * h, r0);
                tmem_ld8(ta + 1 * kOzCols + 8 * h, r1);
                tmem_ld8(ta + 2 * kOzCols + 8 * h, r2);
                tmem_ld8(ta + 3 * kOzCols + 8 * h, r3);
                tmem_ld_wait();
#pragma unroll
                for (int u = 0; u < 8; ++u) {   // |r_o| <= (o + 1) 2^21: both fit 32 bits
                    const int t0 = oz_int(r0[u]) * 256 + oz_int(r1[u]), t1 = oz_int(r2[u]) * 256 + oz_int(r3[u]);
                    V[8 * h + u] = (long long)t0 * 65536 + t1;
                }
                tmem_ld8(ta + 4 * kOzCols + 8 * h, r0);
                tmem_ld8(ta + 5 * kOzCols + 8 * h, r1);
                tmem_ld8(ta + 6 * kOzCols + 8 * h, r2);
                tmem_ld8(ta + 7 * kOzCols + 8 * h, r3);
                tmem_ld_wait();
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const long long lo = (long long)oz_int(r0[u]) * (1 << 24) +
                                         ((long long)oz_int(r1[u]) * 65536 + ((long long)oz_int(r2[u]) * 256 + oz_int(r3[u])));
                    const long long hi = V[8 * h + u] + (lo >> 32);
                    const unsigned w0 = (unsigned)lo, w1 = (unsigned)hi, w2 = (unsigned)(hi >> 32);
                    unsigned k;   // copies of the sign in w2, less one; 30 if it is nothing else
                    asm("bfind.shiftamt.s32 %0, %1;" : "=r"(k) : "r"(w2));
                    k = (k - 1u) & 31u;
                    V[8 * h + u] = (long long)((unsigned long long)__funnelshift_l(w1, w2, k) << 32 | __funnelshift_l(w0, w1, k));
                    ks[h] |= (k & 15u) << (4 * u);
                }
            }
            tc_fence_before();
            mbar_arrive(acc_empty);
            // V 2^(32 - k) in order 7's unit, 2^(56 - 2 (1075 + 10)) times the rows' powers
            if (normal) {
#pragma unroll
                for (int u = 0; u < 32; ++u) {
                    const int sh = ei + __shfl_sync(0xffffffffu, ejl, u) - 2098 - (int)(ks[u / 8] >> (4 * (u % 8)) & 15u);
                    const double v = __longlong_as_double(__double_as_longlong((double)V[u]) + ((long long)sh << 52));
                    sum[u] += V[u] == 0 ? 0.0 : v;
                }
            } else {   // a loop over copies: unrolled, this rare form cost the other 0.8 ms of the 30^3 elasticity step
                long long Vc[32];
                double vc[32];
#pragma unroll
                for (int u = 0; u < 32; ++u) Vc[u] = V[u];
#pragma unroll 1
                for (int u = 0; u < 32; ++u) {
                    const int ej = __shfl_sync(0xffffffffu, ejl, u);
                    const unsigned kw = u < 8 ? ks[0] : u < 16 ? ks[1] : u < 24 ? ks[2] : ks[3];
                    vc[u] = ei == kOzNan || ej == kOzNan ? __longlong_as_double(0x7ff8000000000000ll)
                                                         : oz_value(Vc[u], ei + ej - 2098 - (int)(kw >> (4 * (u % 8)) & 15u));
                }
#pragma unroll
                for (int u = 0; u < 32; ++u) sum[u] += vc[u];
            }
        }
        if (ok && i < d.m) {
            double* C = j0 < d.w ? panel + d.panel_off + (long long)jb * d.ldp + i
                                 : contrib + d.contrib_off + (long long)(jb - d.w) * d.ldc + (i - d.w);
            const long long ld = j0 < d.w ? d.ldp : d.ldc;
#pragma unroll
            for (int u0 = 0; u0 < 32; u0 += 8) {
                double old[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) old[u] = jb + u0 + u < jend && i >= jb + u0 + u ? C[(u0 + u) * ld] : 0.0;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (jb + u0 + u < jend && i >= jb + u0 + u) C[(u0 + u) * ld] = old[u] - sum[u0 + u];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait expired: give copies and MMAs still in flight a bounded time to land before the CTA exits
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 10000000ull) {
        }
    }
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// The tensor-map pair of one front's staging rows: row tiles and column tiles of C.
inline void make_oz_maps(void* l_base, void* w_base, long long rows, int ld, CUtensorMap* out) {
    out[0] = make_region_map(true, l_base, rows, ld, kOzRows);
    out[1] = make_region_map(true, w_base, rows, ld, kOzCols);
}

}  // namespace uchol_dev
