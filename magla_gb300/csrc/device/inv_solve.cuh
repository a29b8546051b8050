// Solves of inverse fronts: fronts of solve_block < w <= inv_cols columns keep
// the whole inverse of the unit-lower triangle of their diagonal block, so that
// a level's solve needs no chain of block solves.  Forward, per front:
//   y_1 = Linv_11 f_1                  (k_fwd_inv_diag: one CTA per block row),
//   f_2 -= L_21 y_1                    (k_fwd_inv_tail: one CTA per chunk of trailing rows);
// backward:
//   g_1 = D^-1 y_1 - L_21^T g_2        (k_bwd_inv_cols: partial sums per chunk of rows, added in
//                                       chunk order by the last chunk of a column block or, of
//                                       large fronts, by k_bwd_inv_reduce),
//   x_1 = Linv_11^T g_1                (k_bwd_inv_diag: one CTA per block column).
// The algebra is the reference's supernodal substitution
// (CAESolvers/UCHOL/UtduNumericFactorization.cs:139-207) with the triangular solve of
// the diagonal block written as a product with its inverse (all but large fronts gather f
// from the children and g_2 from the ancestors where they are read: two launches a level and direction, which
// are what a chain of small fronts waits for); the result differs only
// in rounding.  The inverse is built once per factorisation from the inverses of the
// SB x SB diagonal blocks, by doubling halves: X_21 = -X_22 (L_21 X_11) (k_inv_product).
#pragma once

#include "panel_kernels.cuh"
#include "solve_kernels.cuh"

namespace uchol_dev {

// SB x SB block of the inverse, column-major: (i, i) in the diagonal-block arena, (i, j), i > j,
// in the off-diagonal arena.
template <class Cv, int SB>
__device__ __forceinline__ const Cv* inv_block(const Cv* linv, const Cv* linv_off, int blk, int ob, int i, int j) {
    return i == j ? linv + (long long)(blk + i) * SB * SB
                  : linv_off + ((long long)ob + (long long)i * (i - 1) / 2 + j) * SB * SB;
}

// ---- inversion by halves: one SB x CG strip of a block product sum per CTA ----
//
// What bounds it: few products run at once (a front of nb blocks has at most nb^2 / 4 in a round) and each is long on
// one SM (a 64^3 product takes 66 us on an SM's two FP64 lanes), so a block's columns are dealt out in strips of CG as
// long as that fills the device (launch_inv_product), and the rounds double: 2 log2(nb) launches whose longest sums
// add up to 2 (nb - 1) block products, where building the blocks by diagonals took nb - 1 launches and nb^2 / 2.
// Columns of both operands arrive in chunks of KC rows of B by asynchronous 16-byte copies, the next chunk's under
// the current one's products.
template <class T, int SB, int CG>
struct InvTile {
    static constexpr int V = 16 / (int)sizeof(T);          // elements of a 16-byte load
    static constexpr int OUT = SB * CG / 256;              // outputs of a thread
    static constexpr int TR = OUT >= 64 ? 8 : OUT >= 8 ? 4 : V < OUT ? V : OUT;   // rows of a thread: groups of V, V NX apart
    static constexpr int TC = OUT / TR;
    static constexpr int NX = SB / TR, NY = CG / TC, G = TR / V;
    static constexpr int KC = 128 / (int)sizeof(T);        // rows of B per chunk
    static constexpr int LDB = KC + V;
    static constexpr int kStage = KC * SB + CG * LDB;      // elements of a stage (A chunk, B chunk)
    static constexpr size_t bytes = (size_t)2 * kStage * sizeof(T);
    static_assert(TR % V == 0 && NX * NY == 256, "thread tiles must cover the strip");
};
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}

template <class T, int SB, int CG>
__global__ void __launch_bounds__(256) k_inv_product(const SolveBlockTask* __restrict__ tasks, const SnDev* __restrict__ sn,
                                                     const T* __restrict__ panel, const T* linv, T* linv_off, T* scratch,
                                                     int second) {
    using K = InvTile<T, SB, CG>;
    constexpr int V = K::V, TR = K::TR, TC = K::TC, G = K::G, KC = K::KC;
    extern __shared__ __align__(16) unsigned char inv_smem[];
    T* const sm = reinterpret_cast<T*>(inv_smem);
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = sn[tk.s];
    const int i = tk.k0, j = tk.kn, kb = tk.r1, ke = tk.flags, col0 = blockIdx.y * CG;
    const int tid = threadIdx.x, tx = tid % K::NX, ty = tid / K::NX;
    const T* P = panel + d.panel_off + (long long)i * SB;
    const int rows = min(SB, d.w - i * SB);   // rows of block row i (zero past the front's columns)
    // chunk c: rows [KC c, KC c + KC) of the sum's index, block k = kb + c / (SB / KC)
    auto issue = [&](int c) {
        T* As = sm + (c & 1) * K::kStage;
        T* Bs = As + KC * SB;
        const int k = kb + c / (SB / KC), o = c % (SB / KC) * KC;
        const T* A = second ? inv_block<T, SB>(linv, linv_off, tk.blk, tk.r0, i, k) + o * SB
                            : P + (long long)(k * SB + o) * d.ldp;
        const long long lda = second ? SB : d.ldp;
        const T* B = (second && scratch ? scratch + (long long)(tk.c0 - (i - k) * tk.c1) * SB * SB
                                        : inv_block<T, SB>(linv, linv_off, tk.blk, tk.r0, k, j)) + (long long)col0 * SB + o;
        for (int e = tid; e < KC * SB / V; e += 256) {
            const int r = e % (SB / V) * V, kk = e / (SB / V);
            const int n = second ? V : min(V, max(0, rows - r));
            cp_async16(As + kk * SB + r, n > 0 ? A + r + kk * lda : A, n * (int)sizeof(T));
        }
        for (int e = tid; e < CG * KC / V; e += 256) {
            const int kk = e % (KC / V) * V, c2 = e / (KC / V);
            cp_async16(Bs + c2 * K::LDB + kk, B + (long long)c2 * SB + kk, 16);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    T acc[TC][TR];
#pragma unroll
    for (int q = 0; q < TC; ++q)
#pragma unroll
        for (int u = 0; u < TR; ++u) acc[q][u] = T(0);
    const int nc = (ke - kb) * (SB / KC);
    issue(0);
    for (int c = 0; c < nc; ++c) {
        if (c + 1 < nc) {
            issue(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const T* As = sm + (c & 1) * K::kStage + V * tx;
        const T* Bs = sm + (c & 1) * K::kStage + KC * SB + ty * TC * K::LDB;
#pragma unroll 2
        for (int kk = 0; kk < KC; kk += V) {
            T b[TC][V];
#pragma unroll
            for (int q = 0; q < TC; ++q) *reinterpret_cast<uint4*>(b[q]) = *reinterpret_cast<const uint4*>(Bs + q * K::LDB + kk);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                T a[TR];
#pragma unroll
                for (int g = 0; g < G; ++g)
                    *reinterpret_cast<uint4*>(a + g * V) = *reinterpret_cast<const uint4*>(As + (kk + v) * SB + g * V * K::NX);
                if constexpr (sizeof(T) == 4) {
#pragma unroll
                    for (int q = 0; q < TC; ++q) {
                        const f32x2 bb = pack2(b[q][v], b[q][v]);
#pragma unroll
                        for (int u = 0; u < TR; u += 2) {
                            const f32x2 r = fma2(pack2(a[u], a[u + 1]), bb, pack2(acc[q][u], acc[q][u + 1]));
                            unpack2(r, acc[q][u], acc[q][u + 1]);
                        }
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < TC; ++q)
#pragma unroll
                        for (int u = 0; u < TR; ++u) acc[q][u] += a[u] * b[q][v];
                }
            }
        }
        __syncthreads();   // this stage is refilled by the chunk after next
    }
    // (in place, a CTA has read its strip of T(i, j) by now and no other CTA of the launch reads it)
    T* out = second || !scratch ? linv_off + ((long long)tk.r0 + (long long)i * (i - 1) / 2 + j) * SB * SB
                                : scratch + (long long)tk.c0 * SB * SB;
#pragma unroll
    for (int q = 0; q < TC; ++q)
#pragma unroll
        for (int g = 0; g < G; ++g) {
            T v[V];
#pragma unroll
            for (int u = 0; u < V; ++u) v[u] = second ? -acc[q][g * V + u] : acc[q][g * V + u];
            *reinterpret_cast<uint4*>(out + (long long)(col0 + ty * TC + q) * SB + V * tx + g * V * K::NX) =
                *reinterpret_cast<const uint4*>(v);
        }
}

template <class T, int SB, int CG>
inline void launch_inv_product_cg(const SolveBlockTask* tasks, int count, int second, const SnDev* sn, const T* panel,
                                  const T* linv, T* linv_off, T* scratch, cudaStream_t st) {
    k_inv_product<T, SB, CG><<<dim3(count, SB / CG), 256, InvTile<T, SB, CG>::bytes, st>>>(tasks, sn, panel, linv, linv_off,
                                                                                      scratch, second);
}
// Strip width: whole blocks (the fewest operand reads per product) once they make two CTAs per SM, else the widest
// strips that do, else the narrowest.
template <class T, int SB>
inline void launch_inv_product(const SolveBlockTask* tasks, int count, int second, int sms, const SnDev* sn, const T* panel,
                               const T* linv, T* linv_off, T* scratch, cudaStream_t st) {
    if (count >= 2 * sms) launch_inv_product_cg<T, SB, SB>(tasks, count, second, sn, panel, linv, linv_off, scratch, st);
    else if (4LL * count >= 2 * sms)
        launch_inv_product_cg<T, SB, SB / 4>(tasks, count, second, sn, panel, linv, linv_off, scratch, st);
    else launch_inv_product_cg<T, SB, SB / 8>(tasks, count, second, sn, panel, linv, linv_off, scratch, st);
}

// Shared memory of the inverse-front solve kernels: two SB x SB tile stages, two
// right-hand blocks (SB rows x RG, stride RS) and the partial sums.
template <class T, class Cv, int SB, int RG>
constexpr size_t inv_solve_smem() {
    return (size_t)2 * SB * SB * sizeof(T) + LevelRhs<Cv, SB, RG>::bytes + kLevelSmemSlack;
}

// Register prefetch of an SB x RG right-hand block: thread t holds elements t + 256 q;
// fetch() issues the global loads of the next block before the current tile's products,
// commit() stores them into shared memory (row c at c RS, right-hand side g at + g) after.
template <class Cv, int SB, int RG>
struct RhsPrefetch {
    static constexpr int PQ = (SB * RG + 255) / 256;
    static constexpr int RS = LevelRhs<Cv, SB, RG>::RS;
    Cv v[PQ];
    // f(c, g) -> the value of row c, right-hand side g (zero where absent)
    template <class F>
    __device__ __forceinline__ void fetch(F&& f) {
#pragma unroll
        for (int q = 0; q < PQ; ++q) {
            const int e = (int)threadIdx.x + 256 * q, g = e / SB, c = e - g * SB;
            v[q] = e < SB * RG ? f(c, g) : Cv(0);
        }
    }
    __device__ __forceinline__ void commit(Cv* buf) const {
#pragma unroll
        for (int q = 0; q < PQ; ++q) {
            const int e = (int)threadIdx.x + 256 * q, g = e / SB, c = e - g * SB;
            if (e < SB * RG) buf[c * RS + g] = v[q];
        }
    }
};

// Inverse-diagonal products split in chunks of blocks (plan.hpp, FwdInvDiag): a CTA stores
// the partial sums v of its chunk (row `row`, right-hand sides g0 .. g0+FG-1 of the group) in
// slot slot0 + chunk and counts itself in; the CTA that completes the row's nc chunks adds
// the nc partial sums in chunk order into v and returns true, the others return false.  No
// CTA waits for another.  nc = 1: v is already complete.
template <class Cv, int SB, int FG>
__device__ __forceinline__ bool inv_chunk_combine(Cv (&v)[FG], bool fin, int row, int g0, int ng, int rg, int nrhs,
                                                  int slot0, int chunk, int nc, Cv* __restrict__ pbuf,
                                                  unsigned* __restrict__ cnt) {
    if (nc == 1) return true;
    __shared__ int last;
    if (fin) {
#pragma unroll
        for (int q = 0; q < FG; ++q)
            if (g0 + q < ng) pbuf[((long long)(slot0 + chunk) * nrhs + rg + g0 + q) * SB + row] = v[q];
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* c = cnt + (long long)slot0 * gridDim.y + blockIdx.y;
        last = atomicAdd(c, 1u) == (unsigned)(nc - 1);
        if (last) *c = 0u;   // every chunk has counted in: ready for the next launch
    }
    __syncthreads();
    if (!last) return false;
    if (fin) {
#pragma unroll
        for (int q = 0; q < FG; ++q) {
            Cv s = Cv(0);
            if (g0 + q < ng)
                for (int k = 0; k < nc; ++k) s += __ldcg(&pbuf[((long long)(slot0 + k) * nrhs + rg + g0 + q) * SB + row]);
            v[q] = s;
        }
    }
    return true;
}

// Forward y_i = sum_{j <= i} Linv(i, j) f_j for right-hand sides [RG blockIdx.y, +RG);
// writes y_i (front vector yv).  Thread (row, pid) sums columns [pid CPT, pid CPT + CPT)
// of each block.
template <class T, class Cv, int SB, int RG>
__global__ void __launch_bounds__(256, 1) k_fwd_inv_diag(const SolveBlockTask* __restrict__ tasks, SolveArgs A,
                                                         const Cv* __restrict__ linv, const Cv* __restrict__ linv_off,
                                                         const Cv* __restrict__ fv, Cv* __restrict__ yv,
                                                         const Cv* __restrict__ work, Cv* __restrict__ pbuf,
                                                         unsigned* __restrict__ cnt, int* status) {
    using R = LevelRhs<Cv, SB, RG>;
    constexpr int TPR = R::TP, CPT = SB / TPR, RS = R::RS, FG = R::FG;
    extern __shared__ __align__(128) unsigned char blk_smem[];
    unsigned char* sm = blk_smem + ((1024u - (smem_addr(blk_smem) & 1023u)) & 1023u);
    Cv* const stage0 = reinterpret_cast<Cv*>(sm);        // two Linv tile stages
    auto stage = [&](int k) { return stage0 + k * SB * SB; };
    Cv* const fb0 = stage0 + 2 * SB * SB;                // two blocks f_j: SB rows x RG
    auto fbuf = [&](int k) { return fb0 + k * SB * RS; };
    Cv* part = fb0 + 2 * SB * RS;
    __shared__ unsigned long long bar[2];
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = A.sn[tk.s];
    const int i = tk.k0, ob = tk.r0, blk = tk.blk, j0 = tk.c0, j1 = tk.c1;
    const int rg = blockIdx.y * RG, ng = min(RG, A.nrhs - rg);
    const int tid = threadIdx.x, row = tid % SB, pid = tid / SB;
    const bool fin = RG >= TPR || pid == 0;
    const int g0 = RG >= TPR ? pid * FG : 0;
    const long long fo = A.fvec_off[tk.s];
    if (tid == 0) {
        bar_init(&bar[0]);
        bar_init(&bar[1]);
    }
    constexpr unsigned kTileBytes = SB * SB * sizeof(Cv);
    auto issue = [&](int jj) {
        if (tid == 0) {
            const int st = (jj - j0) & 1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bar_expect(&bar[st], kTileBytes);
            bulk_g2s(stage(st), inv_block<Cv, SB>(linv, linv_off, blk, ob, i, jj), kTileBytes, &bar[st]);
        }
    };
    // f_j, zero past the front's columns and the group's right-hand sides
    RhsPrefetch<Cv, SB, RG> pf;
    auto fetch = [&](int j) {
        pf.fetch([&](int c, int g) {
            const int col = j * SB + c;
            if (g >= ng || col >= d.w) return Cv(0);
            if (RG > 1 && d.m > kGatherRows) return fv[fo + col + (long long)(rg + g) * A.fv_stride];
            return add_children<Cv>(A, fo + col, rg + g, fv, work[d.first_col + col + (long long)(rg + g) * A.ldw]);
        });
    };
    fetch(j0);
    __syncthreads();   // barriers initialised
    issue(j0);
    if (j0 + 1 <= j1) issue(j0 + 1);
    pf.commit(fbuf(0));
    if (j0 + 1 <= j1) fetch(j0 + 1);
    RhsAcc<Cv, RG> acc;
    acc.zero();
    unsigned phase = 0;
    for (int j = j0; j <= j1; ++j) {
        const int st = (j - j0) & 1;
        if (!__syncthreads_and(bar_wait(&bar[st], (phase >> st) & 1u, status))) return;
        phase ^= 1u << st;
        const Cv* tile = stage(st);
        const Cv* fb = fbuf(st);
#pragma unroll 2
        for (int u0 = 0; u0 < CPT; u0 += 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = pid * CPT + u0 + q;
                acc.add(q, tile[row + c * SB], fb + c * RS);
            }
        if (j + 1 <= j1) pf.commit(fbuf(st ^ 1));
        if (j + 2 <= j1) fetch(j + 2);
        __syncthreads();   // the stage is free again
        if (j + 2 <= j1) issue(j + 2);
    }
    acc.store(part + (pid * SB + row) * RG);
    __syncthreads();
    Cv y[FG];
#pragma unroll
    for (int q = 0; q < FG; ++q) {
        const int g = g0 + q;
        y[q] = Cv(0);
        if (fin && g < ng) {
            y[q] = part[row * RG + g];
#pragma unroll
            for (int p = 1; p < TPR; ++p) y[q] += part[(p * SB + row) * RG + g];
        }
    }
    if (!inv_chunk_combine<Cv, SB, FG>(y, fin, row, g0, ng, rg, A.nrhs, tk.r1, j0 / kInvDiagChunk, tk.flags, pbuf,
                                       cnt))
        return;
    if (fin) {
        const int kn = min(SB, d.w - i * SB);
#pragma unroll
        for (int q = 0; q < FG; ++q) {
            const int g = g0 + q;
            if (g >= ng || row >= kn) break;
            const int col = i * SB + row;
            yv[fo + (long long)(rg + g) * A.fv_stride + col] = y[q];
        }
    }
}

// Right-hand sides per CTA of the inverse-front diagonal kernels.
template <class T>
__host__ __device__ constexpr int diag_rhs_group() { return sizeof(T) == 8 ? 4 : 8; }

// Register tiles of the trailing-row kernels.  A thread accumulates RT rows (forward) or
// RT columns (backward) by GT right-hand sides; RT elements are 16 bytes, so the forward
// kernel reads them as one vector.  NG groups of RT rows (columns) cover SB, NH groups of
// GT cover the RG right-hand sides, and the NS remaining thread groups split the half
// tile's columns (forward) or rows (backward); their partial sums are added at the end.
template <class Cv, int SB, int RG>
struct TailTiles {
    static constexpr int RT = 16 / (int)sizeof(Cv);
    static constexpr int GT = RG < 8 ? RG : 8;
    static constexpr int NH = RG / GT;
    static constexpr int NG = SB / RT;
    static constexpr int NS = 256 / (NG * NH);
    static constexpr int RS = LevelRhs<Cv, SB, RG>::RS;   // row stride of the right-hand blocks
    static constexpr int FQ = (SB * RG + 255) / 256;      // results of a thread (forward)
    static_assert(NG * NH * NS == 256 && RG % GT == 0, "thread tiles must cover the CTA");
};

// Shared memory of the trailing-row kernels: two half-tile stages, the transposed half tile
// (backward only; rows of SB + 1 so that the transpose and the column reads are free of
// bank conflicts), two right-hand blocks of SB/2 rows; the partial sums (NS x SB x RG) reuse
// the stages after the last tile.  Two CTAs fit on an SM.
template <class T, class Cv, int SB, int RG, bool kTransposed>
constexpr size_t inv_tail_smem() {
    return (size_t)SB * SB * sizeof(T) + (kTransposed ? (size_t)(SB / 2) * (SB + 1) * sizeof(T) : 0) +
           (size_t)2 * (SB / 2) * TailTiles<Cv, SB, RG>::RS * sizeof(Cv) + kLevelSmemSlack;
}
static_assert((size_t)TailTiles<float, 128, 16>::NS * 128 * 16 * sizeof(float) <= (size_t)128 * 128 * sizeof(float),
              "the partial sums fit in the tile stages");
static_assert((size_t)TailTiles<double, 64, 4>::NS * 64 * 4 * sizeof(double) <= (size_t)64 * 64 * sizeof(double),
              "the partial sums fit in the tile stages");

// Starts a tensor-map tile copy of `bytes` bytes at (x, y) into dst, completing on bar (one thread).
__device__ __forceinline__ void start_box_tile(void* dst, const CUtensorMap* map, int x, int y, unsigned bytes,
                                               unsigned long long* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    bar_expect(bar, bytes);
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// RT consecutive elements of shared memory (16-byte aligned), widened.
__device__ __forceinline__ void lds_vec(const float* p, float (&v)[4]) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
}
__device__ __forceinline__ void lds_vec(const double* p, double (&v)[2]) {
    const double2 q = *reinterpret_cast<const double2*>(p);
    v[0] = q.x;
    v[1] = q.y;
}
// GT values of a right-hand row (16-byte aligned when GT is a multiple of 16 bytes)
template <class Cv, int GT>
__device__ __forceinline__ void lds_rhs(const Cv* p, Cv (&v)[GT]) {
    if constexpr (GT * sizeof(Cv) % 16 == 0) {
#pragma unroll
        for (int g = 0; g < GT; g += 16 / (int)sizeof(Cv)) {
            Cv w[16 / sizeof(Cv)];
            lds_vec(p + g, w);
#pragma unroll
            for (int k = 0; k < 16 / (int)sizeof(Cv); ++k) v[g + k] = w[k];
        }
    } else {
#pragma unroll
        for (int g = 0; g < GT; ++g) v[g] = p[g];
    }
}

// Forward trailing rows [r0, r1) of an inverse front: f = the children's entries - L[r0:r1, 0:w] y, by half tiles
// of SB rows x SB/2 columns (tensor map `maps`: box {SB, SB/2}); the tiles start at r0
// rounded down to 16 bytes.  Thread (row group, right-hand group, column split) keeps an
// RT x GT tile of sums.
template <class T, class Cv, int SB, int RG>
__global__ void __launch_bounds__(256, 2) k_fwd_inv_tail(const SolveBlockTask* __restrict__ tasks, SolveArgs A,
                                                         const CUtensorMap* __restrict__ maps,
                                                         const Cv* __restrict__ yv, Cv* __restrict__ fv, int* status) {
    static_assert(sizeof(T) == sizeof(Cv), "factor and vector elements of one size");
    using W = TailTiles<Cv, SB, RG>;
    constexpr int HC = SB / 2, RT = W::RT, GT = W::GT, NG = W::NG, NH = W::NH, NS = W::NS, RS = W::RS;
    constexpr int CPS = HC / NS;                          // columns of a half tile per split
    constexpr int kAlign = 16 / (int)sizeof(T);
    constexpr unsigned kBytes = SB * HC * sizeof(T);
    extern __shared__ __align__(128) unsigned char blk_smem[];
    unsigned char* sm = blk_smem + ((1024u - (smem_addr(blk_smem) & 1023u)) & 1023u);
    T* const stage0 = reinterpret_cast<T*>(sm);          // two half-tile stages (SB x HC, column-major)
    auto stage = [&](int k) { return stage0 + k * SB * HC; };
    Cv* const yb0 = reinterpret_cast<Cv*>(stage0 + 2 * SB * HC);   // two blocks of y: HC rows x RG
    auto ybuf = [&](int k) { return yb0 + k * HC * RS; };
    Cv* const part = reinterpret_cast<Cv*>(stage0);      // after the last tile: NS x SB x RG
    __shared__ unsigned long long bar[2];
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = A.sn[tk.s];
    const int nh = (d.w + HC - 1) / HC, r0 = tk.r0, r1 = tk.r1, ra = r0 & ~(kAlign - 1);
    const int tid = threadIdx.x, rgp = tid % NG, rh = (tid / NG) % NH, cs = tid / (NG * NH);
    const long long fo = A.fvec_off[tk.s];
    if (tid == 0) {
        bar_init(&bar[0]);
        bar_init(&bar[1]);
    }
    __syncthreads();
    unsigned phase = 0;
    RhsPrefetch<Cv, HC, RG> pf;
    for (int rg = blockIdx.y * RG; rg < A.nrhs; rg += gridDim.y * RG) {
        const int ng = min(RG, A.nrhs - rg);
        auto fetch = [&](int h) {
            const int kn = min(HC, d.w - h * HC);
            pf.fetch([&](int c, int g) {
                return (g < ng && c < kn) ? yv[fo + (long long)(rg + g) * A.fv_stride + h * HC + c] : Cv(0);
            });
        };
        fetch(0);
        if (tid == 0) {
            start_box_tile(stage(0), maps + tk.s, ra, 0, kBytes, &bar[0]);
            if (nh > 1) start_box_tile(stage(1), maps + tk.s, ra, HC, kBytes, &bar[1]);
        }
        Cv f0[W::FQ];   // the children's entries of this thread's results
#pragma unroll
        for (int q = 0; q < W::FQ; ++q) {
            const int e = tid + 256 * q, g = e / SB, i = ra + e - g * SB;
            f0[q] = !(e < SB * RG && g < ng && i >= r0 && i < r1) ? Cv(0)
                    : RG > 1 && d.m > kGatherRows ? fv[fo + i + (long long)(rg + g) * A.fv_stride]
                                              : add_children<Cv>(A, fo + i, rg + g, fv, Cv(0));
        }
        pf.commit(ybuf(0));
        if (nh > 1) fetch(1);
        Cv acc[RT][GT];
#pragma unroll
        for (int a = 0; a < RT; ++a)
#pragma unroll
            for (int g = 0; g < GT; ++g) acc[a][g] = Cv(0);
        for (int h = 0; h < nh; ++h) {
            if (!__syncthreads_and(bar_wait(&bar[h & 1], (phase >> (h & 1)) & 1u, status))) return;
            phase ^= 1u << (h & 1);
            const T* tile = stage(h & 1) + rgp * RT;
            const Cv* yb = ybuf(h & 1) + rh * GT;
#pragma unroll 4
            for (int u = 0; u < CPS; ++u) {
                const int c = cs * CPS + u;
                Cv l[RT], y[GT];
                lds_vec(tile + c * SB, l);
                lds_rhs<Cv, GT>(yb + c * RS, y);
#pragma unroll
                for (int a = 0; a < RT; ++a)
#pragma unroll
                    for (int g = 0; g < GT; ++g) acc[a][g] += l[a] * y[g];
            }
            if (h + 1 < nh) pf.commit(ybuf((h + 1) & 1));
            if (h + 2 < nh) fetch(h + 2);
            __syncthreads();   // the stage is free again
            if (tid == 0 && h + 2 < nh) start_box_tile(stage(h & 1), maps + tk.s, ra, (h + 2) * HC, kBytes, &bar[h & 1]);
        }
        // partial sums of the column splits, then f -= their sum for the chunk's rows
#pragma unroll
        for (int a = 0; a < RT; ++a)
#pragma unroll
            for (int g = 0; g < GT; ++g) part[(cs * SB + rgp * RT + a) * RG + rh * GT + g] = acc[a][g];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < W::FQ; ++q) {
            const int e = tid + 256 * q, g = e / SB, lr = e - g * SB, i = ra + lr;
            if (e >= SB * RG || g >= ng || i < r0 || i >= r1) continue;
            Cv sum = part[lr * RG + g];
#pragma unroll
            for (int p = 1; p < NS; ++p) sum += part[(p * SB + lr) * RG + g];
            fv[fo + (long long)(rg + g) * A.fv_stride + i] = f0[q] - sum;
        }
        __syncthreads();
    }
}

// g = y / D - the nq chunks' partial sums of one column block, in chunk order, for ng right-hand sides: N results a
// thread, the loads of U chunks in flight: the latency of these loads is what the level waits for (23 x 17 x 11
// elasticity, 5 right-hand sides: 28.9 ms with 6 chunks in flight, 29.7 with 2).
template <class Cv, int SB, int N, int U>
__device__ __forceinline__ void add_chunks(const Cv* __restrict__ slot, int nq, const SolveArgs& A, const SnDev& d, int c0,
                                           int ng, long long fo, Cv* __restrict__ fv, const Cv* __restrict__ yv,
                                           const double* __restrict__ diag) {
    const long long step = (long long)A.nrhs * SB;
    long long at[N];
    bool on[N];
    Cv v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int e = threadIdx.x + 256 * k, g = e / SB, col = c0 + e - g * SB;
        on[k] = g < ng && col < d.w;
        at[k] = fo + (long long)g * A.fv_stride + col;
        v[k] = on[k] ? (Cv)((double)yv[at[k]] / diag[d.first_col + col]) : Cv(0);
    }
    for (int q0 = 0; q0 < nq; q0 += U) {
        Cv p[U][N];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < N; ++k)
                p[u][k] = on[k] && q0 + u < nq ? __ldcg(slot + (q0 + u) * step + threadIdx.x + 256 * k) : Cv(0);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (q0 + u < nq) v[k] -= p[u][k];
    }
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (on[k]) fv[at[k]] = v[k];
}

// Backward: column block kb of an inverse front against its trailing rows [r0, r1) (task
// {s, kb, nb, r0, r1, nq, slot}), by half tiles of SB/2 rows x SB columns (tensor map `maps`:
// box {SB/2, SB}), each transposed in shared memory so that a thread's RT columns are read
// without bank conflicts and g is a broadcast.  Thread (column group, right-hand group, row
// split) keeps an RT x GT tile of sums; column group q holds columns q + NG a.  The sums go
// to partial slot `slot` ((slot nrhs + r) SB + c for right-hand side r, column c); the CTA
// that completes the block's chunks (a counter, no waiting) adds them in chunk order into g,
// k_bwd_inv_reduce those of large fronts.
template <class T, class Cv, int SB, int RG>
__global__ void __launch_bounds__(256, 2) k_bwd_inv_cols(const SolveBlockTask* __restrict__ tasks, SolveArgs A,
                                                         const CUtensorMap* __restrict__ maps, Cv* __restrict__ fv,
                                                         const Cv* __restrict__ yv, const double* __restrict__ diag,
                                                         const Cv* __restrict__ work, Cv* __restrict__ partial,
                                                         unsigned* __restrict__ cnt, int* status) {
    static_assert(sizeof(T) == sizeof(Cv), "factor and vector elements of one size");
    using W = TailTiles<Cv, SB, RG>;
    constexpr int HR = SB / 2, RT = W::RT, GT = W::GT, NG = W::NG, NH = W::NH, NS = W::NS, RS = W::RS;
    constexpr int RPS = HR / NS;                          // rows of a half tile per split
    constexpr int TS = SB + 1;                            // row stride of the transposed half tile
    constexpr int kAlign = 16 / (int)sizeof(T);
    constexpr unsigned kBytes = HR * SB * sizeof(T);
    extern __shared__ __align__(128) unsigned char blk_smem[];
    unsigned char* sm = blk_smem + ((1024u - (smem_addr(blk_smem) & 1023u)) & 1023u);
    T* const stage0 = reinterpret_cast<T*>(sm);          // two half-tile stages (HR x SB, column-major)
    auto stage = [&](int k) { return stage0 + k * HR * SB; };
    T* const tt = stage0 + 2 * HR * SB;                   // transposed half tile: row r at r TS
    Cv* const xb0 = reinterpret_cast<Cv*>(tt + HR * TS);  // two blocks of g: HR rows x RG
    auto xbuf = [&](int k) { return xb0 + k * HR * RS; };
    Cv* const part = reinterpret_cast<Cv*>(stage0);      // after the last tile: NS x SB x RG
    __shared__ unsigned long long bar[2];
    __shared__ int last;
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = A.sn[tk.s];
    const int* rows = A.rows + d.rows_off;
    const int kb = tk.k0, r0 = tk.r0, r1 = tk.r1, ra = r0 & ~(kAlign - 1);
    const int ntile = (r1 - ra + HR - 1) / HR;
    const int tid = threadIdx.x, cgp = tid % NG, rh = (tid / NG) % NH, rsp = tid / (NG * NH);
    const long long fo = A.fvec_off[tk.s];
    if (tid == 0) {
        bar_init(&bar[0]);
        bar_init(&bar[1]);
    }
    __syncthreads();
    unsigned phase = 0;
    RhsPrefetch<Cv, HR, RG> pf;
    for (int rg = blockIdx.y * RG; rg < A.nrhs; rg += gridDim.y * RG) {
        const int ng = min(RG, A.nrhs - rg);
        auto fetch = [&](int t) {
            const int tr = ra + t * HR;
            pf.fetch([&](int r, int g) {
                const int gr = tr + r;
                if (g >= ng || gr < r0 || gr >= r1) return Cv(0);
                return RG > 1 && d.m > kGatherRows ? fv[fo + gr + (long long)(rg + g) * A.fv_stride]
                                               : work[rows[gr] + (long long)(rg + g) * A.ldw];
            });
        };
        fetch(0);
        if (tid == 0) {
            start_box_tile(stage(0), maps + tk.s, ra, kb * SB, kBytes, &bar[0]);
            if (ntile > 1) start_box_tile(stage(1), maps + tk.s, ra + HR, kb * SB, kBytes, &bar[1]);
        }
        pf.commit(xbuf(0));
        if (ntile > 1) fetch(1);
        Cv acc[RT][GT];
#pragma unroll
        for (int a = 0; a < RT; ++a)
#pragma unroll
            for (int g = 0; g < GT; ++g) acc[a][g] = Cv(0);
        for (int t = 0; t < ntile; ++t) {
            if (!__syncthreads_and(bar_wait(&bar[t & 1], (phase >> (t & 1)) & 1u, status))) return;
            phase ^= 1u << (t & 1);
            {
                // 16 bytes (RT consecutive rows of one column) per read
                const T* src = stage(t & 1);
                constexpr int QR = HR / RT;   // 16-byte groups per column
                for (int e = tid; e < QR * SB; e += blockDim.x) {
                    const int r = (e % QR) * RT, c = e / QR;
                    T v[RT];
                    lds_vec(src + c * HR + r, v);
#pragma unroll
                    for (int k = 0; k < RT; ++k) tt[(r + k) * TS + c] = v[k];
                }
            }
            __syncthreads();   // tt is ready, the stage is free again
            if (tid == 0 && t + 2 < ntile) start_box_tile(stage(t & 1), maps + tk.s, ra + (t + 2) * HR, kb * SB, kBytes, &bar[t & 1]);
            const Cv* xb = xbuf(t & 1) + rh * GT;
#pragma unroll 4
            for (int u = 0; u < RPS; ++u) {
                const int r = rsp * RPS + u;
                Cv l[RT], x[GT];
#pragma unroll
                for (int a = 0; a < RT; ++a) l[a] = (Cv)tt[r * TS + cgp + NG * a];
                lds_rhs<Cv, GT>(xb + r * RS, x);
#pragma unroll
                for (int a = 0; a < RT; ++a)
#pragma unroll
                    for (int g = 0; g < GT; ++g) acc[a][g] += l[a] * x[g];
            }
            if (t + 1 < ntile) pf.commit(xbuf((t + 1) & 1));
            if (t + 2 < ntile) fetch(t + 2);
            __syncthreads();   // tt and the right-hand block are free again
        }
#pragma unroll
        for (int a = 0; a < RT; ++a)
#pragma unroll
            for (int g = 0; g < GT; ++g) part[(rsp * SB + cgp + NG * a) * RG + rh * GT + g] = acc[a][g];
        __syncthreads();
        for (int e = tid; e < SB * RG; e += blockDim.x) {
            const int g = e / SB, c = e - g * SB;
            if (g >= ng) continue;
            Cv sum = part[c * RG + g];
#pragma unroll
            for (int p = 1; p < NS; ++p) sum += part[(p * SB + c) * RG + g];
            partial[((long long)tk.blk * A.nrhs + rg + g) * SB + c] = sum;
        }
        const int slot0 = tk.c0, nq = tk.c1;
        if (RG > 1 && d.m > kGatherRows) {   // k_bwd_inv_reduce adds the chunks
            __syncthreads();
            continue;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            unsigned* n = cnt + (long long)slot0 * A.nrhs + rg;   // one counter per group of right-hand sides
            last = atomicAdd(n, 1u) == (unsigned)(nq - 1);
            if (last) *n = 0u;   // every chunk has counted in: ready for the next launch
            __threadfence();
        }
        __syncthreads();
        if (!last) continue;
        const Cv* slot = partial + ((long long)slot0 * A.nrhs + rg) * SB;
        const int na = (ng * SB + 255) / 256;   // sums of a thread; about 16 loads in flight
        if (na <= 1) add_chunks<Cv, SB, 1, 16>(slot, nq, A, d, kb * SB, ng, fo + (long long)rg * A.fv_stride, fv, yv, diag);
        else if (na <= 3) add_chunks<Cv, SB, 3, 6>(slot, nq, A, d, kb * SB, ng, fo + (long long)rg * A.fv_stride, fv, yv, diag);
        else add_chunks<Cv, SB, W::FQ, 2>(slot, nq, A, d, kb * SB, ng, fo + (long long)rg * A.fv_stride, fv, yv, diag);
    }
}

// Backward, large fronts: g of column block kb = y / D - its nq partial sums, subtracted in chunk
// order (task {s, kb, nb, slot0, nq, -, -}: the block's chunks have slots slot0 .. slot0+nq-1),
// one CTA per block and right-hand side (blockIdx.y), one thread per column.
template <class Cv, int SB>
__global__ void __launch_bounds__(SB) k_bwd_inv_reduce(const SolveBlockTask* __restrict__ tasks, SolveArgs A,
                                                       Cv* __restrict__ fv, const Cv* __restrict__ yv,
                                                       const double* __restrict__ diag,
                                                       const Cv* __restrict__ partial) {
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = A.sn[tk.s];
    const int kb = tk.k0, slot0 = tk.r0, nq = tk.r1, c = threadIdx.x;
    if (kb * SB + c >= d.w) return;
    for (int r = blockIdx.y; r < A.nrhs; r += gridDim.y) {
        const long long at = A.fvec_off[tk.s] + (long long)r * A.fv_stride + kb * SB + c;
        Cv v = (Cv)((double)yv[at] / diag[d.first_col + kb * SB + c]);
        const Cv* pp = partial + ((long long)slot0 * A.nrhs + r) * SB + c;
        for (int q0 = 0; q0 < nq; q0 += 8) {   // eight loads in flight, subtracted in chunk order
            Cv p8[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) p8[k] = q0 + k < nq ? pp[(long long)(q0 + k) * A.nrhs * SB] : Cv(0);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (q0 + k < nq) v -= p8[k];
        }
        fv[at] = v;
    }
}

// Backward x_j = sum_{i >= j} Linv(i, j)^T g_i (g_i left by k_bwd_inv_cols; y_i / D where the front has no trailing
// rows), right-hand sides [RG blockIdx.y, +RG); writes x_j to the work vector.
template <class T, class Cv, int SB, int RG>
__global__ void __launch_bounds__(256, 1) k_bwd_inv_diag(const SolveBlockTask* __restrict__ tasks, SolveArgs A,
                                                         const Cv* __restrict__ linv, const Cv* __restrict__ linv_off,
                                                         const Cv* __restrict__ fv, const Cv* __restrict__ yv,
                                                         const double* __restrict__ diag, Cv* __restrict__ work,
                                                         Cv* __restrict__ pbuf, unsigned* __restrict__ cnt,
                                                         int* status) {
    using R = LevelRhs<Cv, SB, RG>;
    constexpr int TPC = R::TP, RPT = SB / TPC, RS = R::RS, FG = R::FG;
    extern __shared__ __align__(128) unsigned char blk_smem[];
    unsigned char* sm = blk_smem + ((1024u - (smem_addr(blk_smem) & 1023u)) & 1023u);
    Cv* const stage0 = reinterpret_cast<Cv*>(sm);        // two Linv tile stages
    auto stage = [&](int k) { return stage0 + k * SB * SB; };
    Cv* const gb0 = stage0 + 2 * SB * SB;                // two blocks g_i: SB rows x RG
    auto gbuf = [&](int k) { return gb0 + k * SB * RS; };
    Cv* part = gb0 + 2 * SB * RS;
    __shared__ unsigned long long bar[2];
    const SolveBlockTask tk = tasks[blockIdx.x];
    const SnDev d = A.sn[tk.s];
    const int j = tk.k0, ob = tk.r0, blk = tk.blk, i0 = tk.c0, i1 = tk.c1;
    const int rg = blockIdx.y * RG, ng = min(RG, A.nrhs - rg);
    const int tid = threadIdx.x, ccol = tid % SB, cpart = tid / SB;
    const bool fin = RG >= TPC || cpart == 0;
    const int g0 = RG >= TPC ? cpart * FG : 0;
    const long long fo = A.fvec_off[tk.s];
    if (tid == 0) {
        bar_init(&bar[0]);
        bar_init(&bar[1]);
    }
    constexpr unsigned kTileBytes = SB * SB * sizeof(Cv);
    auto issue = [&](int ii) {
        if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const int st = (ii - i0) & 1;
            bar_expect(&bar[st], kTileBytes);
            bulk_g2s(stage(st), inv_block<Cv, SB>(linv, linv_off, blk, ob, ii, j), kTileBytes, &bar[st]);
        }
    };
    RhsPrefetch<Cv, SB, RG> pf;
    auto fetch = [&](int i) {
        pf.fetch([&](int c, int g) {
            const int col = i * SB + c;
            if (g >= ng || col >= d.w) return Cv(0);
            const long long at = fo + (long long)(rg + g) * A.fv_stride + col;
            return d.m > d.w ? fv[at] : (Cv)((double)yv[at] / diag[d.first_col + col]);
        });
    };
    fetch(i0);
    __syncthreads();   // barriers initialised
    issue(i0);
    if (i0 + 1 <= i1) issue(i0 + 1);
    pf.commit(gbuf(0));
    if (i0 + 1 <= i1) fetch(i0 + 1);
    RhsAcc<Cv, RG> acc;
    acc.zero();
    unsigned phase = 0;
    for (int i = i0; i <= i1; ++i) {
        const int st = (i - i0) & 1;
        if (!__syncthreads_and(bar_wait(&bar[st], (phase >> st) & 1u, status))) return;
        phase ^= 1u << st;
        const Cv* tile = stage(st);
        const Cv* gb = gbuf(st);
#pragma unroll 2
        for (int u0 = 0; u0 < RPT; u0 += 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = cpart * RPT + ((u0 + q + ccol) & (RPT - 1));
                acc.add(q, tile[c + ccol * SB], gb + c * RS);
            }
        if (i + 1 <= i1) pf.commit(gbuf(st ^ 1));
        if (i + 2 <= i1) fetch(i + 2);
        __syncthreads();
        if (i + 2 <= i1) issue(i + 2);
    }
    acc.store(part + (cpart * SB + ccol) * RG);
    __syncthreads();
    Cv x[FG];
#pragma unroll
    for (int q = 0; q < FG; ++q) {
        const int g = g0 + q;
        x[q] = Cv(0);
        if (fin && g < ng) {
            x[q] = part[ccol * RG + g];
#pragma unroll
            for (int p = 1; p < TPC; ++p) x[q] += part[(p * SB + ccol) * RG + g];
        }
    }
    if (!inv_chunk_combine<Cv, SB, FG>(x, fin, ccol, g0, ng, rg, A.nrhs, tk.r1, (i0 - j) / kInvDiagChunk, tk.flags,
                                       pbuf, cnt))
        return;
    if (fin) {
        const int kn = min(SB, d.w - j * SB);
#pragma unroll
        for (int q = 0; q < FG; ++q) {
            const int g = g0 + q;
            if (g >= ng || ccol >= kn) break;
            work[d.first_col + j * SB + ccol + (long long)(rg + g) * A.ldw] = x[q];
        }
    }
}

}  // namespace uchol_dev
