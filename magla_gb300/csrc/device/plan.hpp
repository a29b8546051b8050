// Host-side execution plan of the device numeric phase: tree levels, memory
// layout of fronts, and the task lists every kernel launch consumes.  Built
// once per (symbolic pattern, block configuration) and reused by every
// factorisation and solve.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "common.cuh"

namespace uchol_dev {

constexpr int kTailRowsPlan = 1024;  // trailing rows per forward tail task, mixed path
constexpr int kTailRowsPlan64 = 128; // and FP64 (its products hold the SM's FP64 pipe: 2 us at 64 columns)
constexpr int kColRowsPlan = 2048;   // trailing rows per backward column-dot task (longer columns: partial sums)
constexpr int kColRowsPlan64 = 1024; // and FP64
constexpr int kInvColRowsPlan = 1024;   // trailing rows per backward partial-sum task of an inverse front
// Widest front whose diagonal block is kept inverted for the solves.  The inverse costs w^3 / 3 operations per
// factorisation and saves a chain of w / SB block solves (about 9 us each in the mixed path) per solve and direction.
// FP32, factorisation / one application of the factor to 1, 4 and 16 right-hand sides in ms, by the widest inverse:
//   40^3 elasticity, contrast 1e4   2048: 27.6 / 3.22 7.47 10.5   4096: 28.6 / 2.87 6.26 8.99   8192: 33.6 / 2.02 3.72 6.08
//   30^3 elasticity, BF16           2048: 38.4 / 4.16 9.67 12.6   4096: 39.2 / 3.93 9.00 11.8   8192: 40.4 / 3.65 8.09 10.7
//                                   16384: 66.3 / 2.28 4.01 6.23
// 8192 pays from five applications a factorisation on with one right-hand side and from two with several; refined solves
// make five to ten (40^3 contrast 62.5 -> 58.0 ms a step, 30^3 BF16 78.1 -> 76.2).  16384 would take nineteen.  A caller of
// fewer applications sets the option to 2048 (40^3, one: 30.8 ms against 35.6).  FP64, where the pipe does 1.2 TFLOP/s and one
// application is usual: 4096 columns cost 20 ms more on 30^3 elasticity (84 -> 105 ms).
constexpr int kDefaultInvCols = 8192;     // mixed path
constexpr int kDefaultInvCols64 = 2048;   // FP64
constexpr int kOzBlock = 128;         // FP64 tensor-core updates: columns of an outer block (one chunk of digits)
// Fewest rows of a front that takes them.  Refactorisation plus solve, fronts from this size / the FP64 pipe for all:
// elasticity 30^3 84 / 539 ms, 20^3 20.1 / 53.9, 14^3 7.3 / 10.2, one modulus 12^3 5.4 / 6.8; from 1024 rows 3 to 7%
// slower than from 384, and below 384 the difference is within 2%.
constexpr int kOzMinRows = 384;
constexpr int kSuperBlocks = 4;       // tensor-core path: outer blocks per super-block of the own-column updates
constexpr int kDefaultMergeCols = 2048;   // widest device front made of a chain of supernodes (merge_chains)
constexpr int kInvWarpCols = 32;         // widest diagonal block inverted by one warp
constexpr int kInvDiagChunk = 2;         // inverse blocks per task of the inverse-front diagonal products

struct PlanConfig {
    int pivot_block = 32;     // FP64 pivot block (the reference's PanelWidth)
    int outer_block = 32;     // Schur-update block (== pivot_block on the FP64 path)
    int small_mask = 0x7;     // bit b: fronts with 32b < m <= 32(b+1) are factorised by one CTA in shared memory
    bool tensor_core = false; // outer updates on tcgen05 from staged operands
    int solve_block = 64;     // column block of the triangular solves
    int inv_cols = 0;         // > 0: fronts of solve_block < w <= inv_cols columns keep the whole inverse of their
                              // unit-lower diagonal block, and their solves run without a block chain
    int merge_cols = 0;       // > 0: single-child chains of supernodes grouped into device fronts of at most
                              // this many columns (see merge_chains); 0: one device front per supernode
    double merge_fill = 0.05; // largest growth of the stored entries a grouping may cost
    bool side_extend_add = false;   // tensor-core path: the extend-add into the contribution columns of
                                    // large fronts runs on a second stream, beside the level's outer blocks
    int oz_rows = 0;                // FP64 path, > 0: fronts of at least this many rows take their updates on the tensor
                                    // cores, from digit slices (oz_gemm.cuh)
    bool inv_in_place = false;      // the inversion's intermediate products take their results' place, not a scratch arena
    bool gather_lists = true;       // forward solves read the children's entries as they go, from lists of them
    int sms = 0;                    // > 0: the device's SM count (sizes the backward inverse-front chunks)
};

// Device fronts from the supernode partition: runs of supernodes in which each
// one is the only child of the next are grouped into one front, as long as the
// group stays within cfg.merge_cols columns and its lower-trapezoid entries
// exceed the members' own by at most cfg.merge_fill.  A group's rows are its
// columns followed by the last member's trailing rows (every earlier member's
// trailing rows outside the group are among them), so the group is a valid
// front of the same elimination order: the entries it adds are structural zeros
// that stay exactly zero, and its parent's front contains its trailing rows.
struct FrontStructure {
    int count = 0;
    std::vector<int> first_column, parent, child_ptr, children, front_ptr, front_rows;
    std::vector<int> group_of;   // per supernode: its device front
};
FrontStructure merge_chains(int n, int count, const int* first_column, const int* parent, const int* child_ptr,
                            const int* children, const int* front_ptr, const int* front_rows, int max_cols,
                            double max_fill);

// One kernel launch: a contiguous range of tasks in one of the task arrays.
struct Launch {
    enum Kind : int {
        ExtendAdd, SmallFronts, PivotBlock, Trsm, SimtUpdate, TcUpdate, DiagBlock, PanelSolve, OzSlice,
        KindCount
    } kind;
    int begin, count;   // task range
    long long tiles;    // update launches: total tiles (= grid size)
    int variant = 0;    // SmallFronts: lanes per front (8, 16, 32) or 0 (a CTA each); SimtUpdate: tile edge (16 or 32);
                        // TcUpdate: rows of a tile (64, 128, 256); PanelSolve: the same (64, 128)
    int stream = 0;     // 0: main stream; 1: side stream, forked from the main stream at this point;
                        // 2: main stream after joining the side stream
};

struct SolveLaunch {
    enum Kind : int {
        FwdGather, FwdSolo, FwdLevel, BwdGather, BwdTail, BwdSolo, BwdLevel, FwdTail, BwdTailReduce,
        FwdInvDiag, FwdInvTail, BwdInvCols, BwdInvDiag, BwdInvReduce, KindCount
    } kind;
    int begin, count;   // tasks; level launches: the chains (one per front)
    int steps;          // level launches: most diagonal blocks of one front of the level
    int bulk_begin, bulk_count;   // level launches: the bulk chunks
    int progress_off;             // level launches: first progress counter of the bulk chunks
    long long chain_work, bulk_work;   // level launches: block solves and chunk updates (CTA split)
    int long_chains;                   // level launches: fronts of three or more diagonal blocks
    int ndiag;                         // level launches: bulk chunks [0, ndiag) are diagonal blocks
    long long diag_work;               // level launches: chunk updates of those
    int large = 0;                     // gathers and reductions of large inverse fronts: not for one right-hand side
};

// Inverse fronts (cfg.inv_cols): the off-diagonal blocks (i, j), i > j, of the
// inverse of the unit-lower diagonal block, SB x SB column-major each, front s's
// at block index ob_s + i (i - 1) / 2 + j of the off-diagonal arena.  Tasks:
//   inversion            {s, i, j, ob_s, k0, k1, blk, t, z}: by halves.  A group of 2 z blocks whose two halves
//                        are inverted gets its off-diagonal half X_IJ = -X_II (L_IJ X_JJ): first
//                        T(i, j) = sum_{k0 <= k < k1} L(i, k) X(k, j), T's block at index t of the scratch arena
//                        (T(k, j) at t - (i - k) z), then X(i, j) = -sum_{k0 <= k < k1} X(i, k) T(k, j).  In place
//                        (cfg.inv_in_place), T(i, j) is where X(i, j) will be, and the second products take a launch
//                        per block row of the halves, the last row first: row i reads T(k, j), k <= i;
//   FwdInvDiag           {s, i, nb, ob_s, slot0, nc, blk, j0, j1}: the part j0 <= j <= j1 of
//                        y_i = sum_{j <= i} Linv(i, j) f_j (f gathered from the children as it is read); block row i
//                        is split in nc chunks of kInvDiagChunk blocks (partial slots slot0 .. slot0+nc-1; nc = 1: no
//                        split);
//   FwdInvTail           {s, -, nb, r0, r1, -, -}: f[r0, r1) = the children's entries - L[r0:r1, 0:w] y;
//   BwdInvCols           {s, kb, nb, r0, r1, -, slot, slot0, nq}: partial sums of L[r0:r1, block kb]^T g
//                        into partial slot `slot` (the block's nq chunks have slots slot0 .. slot0+nq-1); the last of
//                        them to be done writes g = y / D - their sum of the block's columns, unless the front is
//                        large (more than kGatherRows rows, several right-hand sides);
//   BwdInvReduce         {s, kb, nb, slot0, nq, -, -}: that sum for large fronts;
//   BwdInvDiag           {s, j, nb, ob_s, slot0, nc, blk, i0, i1}: the part i0 <= i <= i1 of
//                        x_j = sum_{i >= j} Linv(i, j)^T g_i, in chunks as FwdInvDiag.
// blk is the diagonal-inverse index of the front's block 0.
//
// Inverse fronts read the children's and the ancestors' entries inside their kernels and the last chunk of a column
// block adds its partial sums; a level then has four launches, not seven, which bounds chains of small fronts (24^3 x 3
// grid, FP64, 33 right-hand sides: 7.53 -> 7.16 ms; 20^3 elasticity with one is the same within its noise, 1.02 ms).  Every
// block row and column of a front reads the entries again, which costs more the wider the front is and the more right-hand
// sides there are; fronts of more than kGatherRows rows are gathered and reduced by launches of their own.  One application
// in ms with those launches for every front / as here / for none, by right-hand sides:
//   60 x 60 x 30 elasticity, natural order   2: 27.2 / 27.2 / 25.4   4: 28.6 / 28.6 / 27.9   8: 29.8 / 29.9 / 32.2   16: 32.7 / 32.9 / 37.4
//   40 x 40 x 20 elasticity, natural order   2: 12.7 / 12.7 / 11.4   8: 14.0 / 14.1 / 16.2   16: 14.9 / 15.0 / 18.7
//   30^3 elasticity, AMD                     2: 2.03 / 1.99 / 1.91   4: 2.25 / 2.24 / 2.19   8: 2.56 / 2.64 / 2.64   16: 3.17 / 3.33 / 3.38
// (2048 rows: as the first on the natural orders, as here on 30^3; 8192: as the last, but 27.1, 28.6, 30.1 and 33.2 on the
// first mesh.)  So 4096 is within 5% of the better side from 8 right-hand sides on and gives up 4 to 11% at 2: the number of
// right-hand sides matters more than the rows.
// One right-hand side gains without them (40^3 elasticity, contrast 1e4: 53.2 -> 52.6 ms; 30^3 BF16 70.3 -> 69.8 ms), so
// its solves leave those launches out.
constexpr int kGatherRows = 4096;

struct InvLaunch {
    int begin, count;   // inversion tasks
    int second;         // 0: T = L X, 1: X = -X T
};

// Solve task of supernode s.  Gathers: rows [r0, r1) of the front vector.
// Level launches: a chain (k0 = bulk index of the chunk of the front's
// diagonal block 0, blk = its first diagonal block) or a bulk chunk of rows
// (forward) or own columns (backward) [r0, r1) (blk as for chains).
// Trailing-row dots: columns [k0, k0+kn) against rows [r0, r1).  Inversion:
// diagonal block [k0, k0+kn), blk = its index in the inverse arena.
struct SolveBlockTask {
    int s, k0, kn, r0, r1;
    int flags, blk;
    int c0 = 0, c1 = 0;   // inverse-front diagonal tasks: the range of inverse blocks summed; BwdInvCols: slot0, nq
};

// Host mirror of the device TcJob (tc_gemm.cuh): one rank-kn update of a front.
struct TcJobHost {
    long long tile_begin;
    int s, c0, cend, kbeg, kn, map;
};

// Front-size buckets of the one-CTA small-front kernel: 32 rows each, up to kSmallFrontLimit
// rows (the whole front in FP64 shared memory: 160^2 * 8 bytes = 200 KB).
constexpr int kSmallBucketRows = 32;
constexpr int kSmallFrontLimit = 160;
constexpr int kSmallBuckets = kSmallFrontLimit / kSmallBucketRows;
inline bool small_front(const PlanConfig& cfg, int m) {
    return m <= kSmallFrontLimit && ((cfg.small_mask >> ((m - 1) / kSmallBucketRows)) & 1);
}

// Rows in 16 bytes of the factor storage type (float on the tensor-core path, else double):
// tile copies by tensor map must start on a multiple of it.
inline int kTileAlignRows(const PlanConfig& cfg) { return cfg.tensor_core ? 4 : 2; }

struct Plan {
    PlanConfig cfg;
    int n = 0, count = 0, levels = 0;          // count: device fronts
    int supernodes = 0;                        // supernodes of the symbolic partition
    std::vector<int> front_rows, child_ptr, children;   // structure of the device fronts (solves)
    std::vector<int> level_of;                 // per supernode
    std::vector<SnDev> sn;                     // per supernode
    std::vector<int> rel;                      // parent-local index of each trailing row
    std::vector<long long> assemble_pos;       // per matrix value: offset in the factor arena
    long long factor_elems = 0;                // panels
    long long contrib_elems = 0;               // contribution arena (planned peak)
    long long fvec_elems = 0;                  // front-vector workspace of the solves (per RHS)
    std::vector<long long> fvec_off;           // per supernode offset into the front-vector workspace

    // factorisation tasks
    std::vector<EaItem> ea_items;
    std::vector<EaEntry> ea_entries;
    std::vector<int> small_fronts;
    std::vector<PanelTask> pivot_tasks;   // one per (front, pivot block); mixed path: per (front, outer block)
    std::vector<PanelTask> panel_tasks;   // TRSM / panel-solve row chunks
    int diag_slots = 0;                   // mixed path: most diagonal blocks of one launch (inverse workspace slots)
    double panel_flops = 0.0;             // mixed path: flops of the panel-solve products
    std::vector<UpdJob> simt_jobs;
    std::vector<TcJobHost> tc_jobs;
    std::vector<StageInfo> stage;              // per supernode (tensor-core path)
    std::vector<int> map_front;                // front of each tensor-map pair
    std::vector<Launch> launches;
    int max_small_m = 0;                  // of the fronts taken by a CTA each
    long long stage_elems = 0;                 // elements of each operand staging arena (tensor-core path; FP64: digits)
    long long oz_exps = 0;                     // row exponents of a level (FP64 tensor-core updates)
    double tc_flops = 0.0;                     // algorithmic flops of the tensor-core updates (lower triangle)
    double simt_flops = 0.0;                   // algorithmic flops of the SIMT updates

    // solve tasks
    std::vector<unsigned> gather_ptr;          // per position of the front vectors: its entries of gather_src
    std::vector<unsigned> gather_src;          // front-vector positions of the children's update entries, in child order
                                               // (both empty: every front's vector is gathered by a launch)
    std::vector<SolveBlockTask> solve_tasks;
    std::vector<SolveBlockTask> inv_blocks;    // every diagonal block, for the inversion after a factorisation
    std::vector<SolveLaunch> fwd_launches, bwd_launches;
    std::vector<SolveBlockTask> inv_warp, inv_cta;   // those the factorisation kernels do not invert themselves: up to
                                               // kInvWarpCols columns (a warp each), wider (a CTA each)
    std::vector<int> front_blk;                // per front: index of its first diagonal block
    std::vector<SolveBlockTask> inv_tasks;     // inverse fronts: off-diagonal inverse blocks, by doubling halves
    std::vector<InvLaunch> inv_launches;
    long long inv_off_blocks = 0;              // blocks of the off-diagonal inverse arena
    long long inv_scratch_blocks = 0;          // blocks of the inversion's scratch (T of one round)
    int inv_partial_slots = 0;                 // most BwdInvCols partial slots of one launch (SB x nrhs each)
    int inv_diag_slots = 0;                    // most inverse-diagonal partial slots of one launch (SB x nrhs each)
    int progress_count = 0;                    // progress counters of all level launches
    int bwd_partial_slots = 0;                 // most backward column-dot partial slots of one launch (8 x nrhs each)
};

// Algorithmic flops (2 per multiply-add, lower triangle) and tiles of an update job.
double job_flops(const UpdJob& J, const SnDev& d);
long long job_tiles(const UpdJob& J, const SnDev& d, int T);

// Throws std::runtime_error on inconsistent symbolic input.
Plan build_plan(int n, int count, const int* first_column, const int* parent, const int* child_ptr,
                const int* children, const int* front_ptr, const int* front_rows, const int* diag_value_index,
                const int* pattern_ptr, const int* pattern_rows, const int* lower_start, const int* lower_value_ptr,
                const int* lower_value_index, int nnz, const PlanConfig& cfg);

}  // namespace uchol_dev
