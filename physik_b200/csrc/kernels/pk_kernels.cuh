// pk_kernels.cuh -- device-side views and launchers shared by the kernel and ABI
// translation units.  Everything here is internal to libpkcuda.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pk_math.cuh"
#include "pk_res_plan.h"
#include "pk_slab_plan.h"

namespace pk {

// Step flags (mirrored in include/pkcuda.h as PK_FLAG_*).
enum : unsigned {
    kFlagPrecomputeFailed = 0x1u,
    kFlagSingularDiag = 0x2u,
    kFlagInvalidRhs = 0x4u,
    kFlagBreakdown = 0x8u,
    kFlagNonFiniteDv = 0x10u,
    kFlagIntegrateAbort = 0x20u,
    kFlagPolarIdentity = 0x40u,
    kFlagPolarFp64 = 0x80u,
    kFlagBarrierTimeout = 0x100u,
    kFlagRowTooLong = 0x200u,
    kFlagSolved = 0x1000u,
    kFlagIntegrated = 0x2000u,
    kFlagConverged = 0x4000u,
    kFlagRefinedFp64 = 0x8000u,
};

struct GridSync {
    unsigned arrive;
    unsigned gen;
    int err;
    int pad;
};

struct DevStats {
    int iterations;
    int converged;
    double residual_norm;
    unsigned flags;
    int polar_fp64_count;
    int polar_identity_count;
    unsigned batch_missing;  // batched solve: success flags some body lacks
};

// Upper-stored symmetric BSR plus its transpose index: for row r, the blocks (c, r)
// with c < r are lt_block[lt_start[r] .. lt_start[r+1]) and c = lt_row[...].
template <class Real>
struct BsrView {
    int n;
    const int* row_start;
    const int* col;
    const Real* values;  // 9 per block, column-major
    const int* lt_start;
    const int* lt_row;
    const int* lt_block;
};

template <class Real>
struct TetView {
    int tet_count;
    const int4* nodes;               // world node ids
    const unsigned char* enabled;    // bit 0: active, rest volume > 0, body simulated; bit 1: linear FEM
    const Real* dm_inv;              // 9 per tet, column-major
    const Real* params;              // 4 per tet: rest volume, lambda, mu, damping
    // tet_rec() values per tet, written by the tet kernel each step and read by the row
    // kernels (one aligned record per tet): four corners of four values P_k = sqrt(V mu) R g_k
    // and lambda / mu, then four of B_k and 0, with B_k = T g_k - dt c v_k the tet's right-hand
    // side at corner k (T = -(dt S + dt^2 Q), S = R V sigma, Q g_a the tet's sum_b K_ab v_b); in
    // FP64 then V mu g_a.g_b (10) and R R^T (6).  A tet that is not folded so has NaN in place
    // of every lambda / mu, and its form in place of B_0's 0: kFormForces, B_k = -S g_k (lambda
    // / mu in place of the other zeros); kFormPlain (blocks that might overflow, V mu too small
    // for its root, lambda / mu too large, or in FP32 a rotation whose iteration ran out), R in
    // the first three corners and S in the next three; kFormSkip, no part in this step.
    // Explicit step: kTetForces values per tet, four corners of the force -S g_k and the damping.
    Real* rec;
    const Real* rest;                // 12 per tet: DmInv, rest volume, lambda, mu (launch_tet_pack)
};
template <class Real>
constexpr int tet_rec()
{
    return sizeof(Real) == 4 ? 32 : 48;
}
constexpr int kTetForces = 16;
constexpr int kFormForces = 1, kFormPlain = 2, kFormSkip = 3;

template <class Real>
struct AssemblyArgs {
    TetView<Real> tets;
    BsrView<Real> a;
    int node_count;
    const int* dyn_to_node;
    const int* node_to_dyn;
    const Real* mass;                // per world node
    const Real* x;                   // 3 per world node
    Real* v;                         // 3 per world node (written only in explicit mode)
    Real* x_out;                     // explicit mode position update target
    const int* inc_start;            // per dyn row
    const int* inc_list;             // t*4 + a
    // The blocks' tets (block_list_kernel); NULL: one thread per row over its incidences.
    int nnz;
    const int2* blk_range;           // per stored block
    const unsigned* blk_list;
    const int* blk_missing;          // rows whose tets couple a block the pattern lacks
    int fold;                        // fold the tets' K v into their right-hand sides
    Real* values;                    // out: A blocks
    Real* rhs;                       // out: b
    Real* minv;                      // out: block-Jacobi inverse
    Real dt;
    Real gravity[3];
    int use_jacobi;
    int linear;
    int explicit_mode;
    unsigned* flags;
    DevStats* stats;
    // Transient point connections (PointConnection::UpdateSystem); conn_inc_start is
    // NULL when there are none.
    int conn_count;
    const int4* conn_nodes;          // 4 world nodes per connection
    const Real* conn_params;         // kConnParams per connection: weights (4), target (3), stiffness, damping
    Real* conn_eval;                 // 4 per connection: its force (3) and 1 when it applies this step, else 0
    const int* conn_inc_start;       // per dyn row
    const int* conn_inc_list;        // connection*4 + corner (corners with a non-zero weight)
    // Host-emitted stiffness blocks and forces (SolverData::AddStiffnessBlock / AddNodeForce
    // from custom components); ext_rhs_start is NULL when there are none.
    const Real* ext_blocks;          // 9 per block, column-major
    const int2* ext_nodes;           // per block: its row node and column node
    const int* ext_rhs_start;        // per dyn row: blocks whose row node is that row (rhs -dt^2 B v_col)
    const int* ext_rhs_list;
    const int* ext_mat_start;        // per dyn row: blocks it holds in its upper row
    const int* ext_mat_list;         // block index, | 0x80000000 when the transpose is added
    const Real* ext_force;           // 3 per dyn row, or NULL
};
constexpr int kConnParams = 9;

template <class Real, class Acc>
struct PcgArgs {
    BsrView<Real> a;
    const Real* b;
    const Real* minv;
    Real* x;
    Real* r;
    // Search-direction records, 8 values per row {s.x, s.y, s.z, 0, d.x, d.y, d.z, 0}
    // (32-byte aligned for float), ping-ponged between iterations so a neighbour's
    // s + beta*d is one 256-bit load.
    Real* sd0;
    Real* sd1;
    Real* q;
    Acc* part_a;      // [grid]
    Acc* part_b;      // [grid * 2]
    int* part_bad;    // [grid * 4]: phase A, init/phase B, final check
    GridSync* sync;
    int max_iterations;
    Acc tolerance;
    int skip_on_flags;     // skip the solve when assembly flagged failure
    int integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
    unsigned* flags;
    DevStats* stats;
    // SpMV tiles staged into shared memory by TMA bulk copies, 8 ints per tile:
    // {first row, end row, rs0, row words, k0, blocks, e0, transpose entries}, each range
    // widened to 16-byte boundaries; ntiles == 0 selects the unstaged SpMV.
    int ntiles;
    const int* tile_desc;
};

// Shared-memory tile of the staged SpMV: at most kTileRowCap row_start / lt_start
// entries, kTileCapU upper blocks (values + columns) and kTileCapL transpose entries,
// each range widened to 16-byte boundaries for the bulk copies.
constexpr int kTileRowsMax = 64;
constexpr int kTileRowCap = kTileRowsMax + 8;
constexpr int kTileCapU = 576;
constexpr int kTileCapL = 512;
template <class Real>
constexpr size_t tile_buffer_bytes()
{
    return size_t(2 * kTileRowCap) * 4 + size_t(kTileCapU) * 9 * sizeof(Real) + size_t(kTileCapU) * 4 +
           size_t(2 * kTileCapL) * 4;
}

// ------------------------------------------------------------------ ring-staged PCG
// The ring-staged PCG kernel (pk_pcg_ring.cu) cuts the rows into tiles of at most kRows
// consecutive rows and streams each tile's part of the matrix -- row extents, upper
// blocks with their columns, and the transposed index (rows and block numbers of the
// lower entries) -- into shared memory with TMA bulk copies, through a ring of kStages
// buffers filled by one producer warp.  Consumer warps, in kRingGroups groups that take
// every kRingGroups-th ring position, compute the tile's rows of q = A (s + beta d)
// from the staged data plus gathers of the neighbours' {s, d} records and of the
// transposed lower blocks (both L2 hits, as the grid sweeps one wavefront through the
// matrix).  kStages is a multiple of kRingGroups, so a stage is always reused by the
// group that used it last and its mbarrier parity cannot be mistaken.
// Caps are in entries; every span is widened to 16-byte boundaries (row words to 4,
// blocks and lower entries to 4).
template <class Real>
struct RingTile;
template <>
struct RingTile<float> {
    static constexpr int kRows = 32, kRsCap = 40, kCapU = 320, kCapL = 288;
    static constexpr int kStages = 12, kLanesPerRow = 4;  // 32 rows per consumer group of 4 warps (4 stages each)
};
template <>
struct RingTile<double> {
    static constexpr int kRows = 16, kRsCap = 24, kCapU = 160, kCapL = 144;
    static constexpr int kStages = 12, kLanesPerRow = 8;  // 16 rows per consumer group of 4 warps
};
constexpr int kRingGroups = 3;  // 13 warps: at most 4 per SM sub-partition, so 128 registers
constexpr int kRingGroupWarps = 4;
constexpr int kRingConsumerWarps = kRingGroups * kRingGroupWarps;
constexpr int kRingThreads = 32 * (kRingConsumerWarps + 1);  // + one producer warp
constexpr int kRingDescInts = 8;  // per tile: ra, rb, rs0, nrs, k0, nk, e0, ne
constexpr int kRingMaxTilesPerBlock = 512;

constexpr size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Byte offsets of one ring stage, then of the block's descriptor table after the ring.
template <class Real>
struct RingLayout {
    using T = RingTile<Real>;
    static constexpr size_t kRs = 0;
    static constexpr size_t kLts = kRs + 4 * T::kRsCap;
    static constexpr size_t kVals = align_up(kLts + 4 * T::kRsCap, 16);
    static constexpr size_t kCol = align_up(kVals + sizeof(Real) * 9 * T::kCapU, 16);
    static constexpr size_t kLtr = align_up(kCol + 4 * T::kCapU, 16);
    static constexpr size_t kLtb = align_up(kLtr + 4 * T::kCapL, 16);
    static constexpr size_t kBytes = align_up(kLtb + 4 * T::kCapL, 128);
    static constexpr size_t kTable = kBytes * T::kStages;
    static constexpr size_t kTotal = kTable + 4 * kRingDescInts * size_t(kRingMaxTilesPerBlock);
};

// One block's published partials for a grid exchange (double buffered by generation).
struct __align__(32) ExSlot {
    double v0, v1;
    int bad;
    unsigned gen;
    int pad0, pad1;
};

template <class Real, class Acc>
struct RingPcgArgs {
    BsrView<Real> a;
    int nnz;                     // stored upper blocks
    int ntiles;
    const int* desc;             // kRingDescInts per tile
    const Real* b;
    const Real* minv;
    Real* x;
    Real* r;
    Real* sd0;                   // {s.xyz, 0, d.xyz, 0} per row, ping-ponged
    Real* sd1;
    Real* q4;                    // {q.xyz, 0} per row
    ExSlot* slots;               // [2][grid]
    GridSync* sync;              // err flag
    int max_iterations;
    Acc tolerance;
    int skip_on_flags;
    int integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
    unsigned* flags;
    DevStats* stats;
};

// ------------------------------------------------------------------ batched PCG
// Batched per-body solve (pk_pcg_batch.cu).  parts: 8 ints per block {body, first row,
// end row, index in the body's group, first block of the group, group size, 0, 0}.
constexpr int kBatchThreads = 256;

struct BatchBodyStats {
    int iterations;
    int converged;
    double residual_norm;
    unsigned flags;
    int pad;
};

template <class Real, class Acc>
struct BatchPcgArgs {
    BsrView<Real> a;
    int nnz;
    const int* parts;
    const Real* b;
    const Real* minv;
    Real* x;
    Real* r;
    Real* sd0;
    Real* sd1;
    Real* q4;
    ExSlot* slots;   // [2][grid]
    GridSync* sync;  // err flag
    int max_iterations;
    Acc tolerance;
    int skip_on_flags;
    int integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
    unsigned* flags;
    unsigned* missing;
    DevStats* stats;
    BatchBodyStats* body_stats;
};

// ------------------------------------------------------------------ part-resident PCG
// The part-resident ("slab") PCG kernel (pk_pcg_slab.cu; layout in pk_slab_plan.h): one
// block per part, FP32 storage.  Shared memory: the window's search directions
// (kSlabWinCap x 3 floats), the ring of kSlabStages tile stages, the part's tile table,
// and for the symmetric stream form the consumer groups' transposed-product rings.
constexpr int kSlabGroupWarps = 4;
constexpr int kSlabConsumerWarps = kSlabGroups * kSlabGroupWarps;
// + one producer warp (the stream) and one halo warp (the window's halo rows, while the
// consumers stream the part's interior tiles)
constexpr int kSlabThreads = 32 * (kSlabConsumerWarps + 2);
constexpr size_t kSlabWinBytes = 12 * size_t(kSlabWinCap);
constexpr size_t kSlabRingOffset = kSlabWinBytes;
constexpr size_t kSlabTableOffset = kSlabRingOffset + size_t(kSlabStages) * kSlabStageBytes;
constexpr size_t kSlabFullSmemBytes = kSlabTableOffset + 16 * size_t(kSlabMaxTiles);
constexpr size_t kSlabSymTableOffset = kSlabRingOffset + size_t(kSlabStages) * kSymStageBytes;
constexpr size_t kSlabSymTpOffset = kSlabSymTableOffset + 16 * size_t(kSlabMaxTiles);
constexpr size_t kSlabSymSmemBytes = kSlabSymTpOffset + 12 * size_t(kSlabGroups) * kSymRingSlots;
constexpr size_t kSlabSmemBytes = kSlabFullSmemBytes > kSlabSymSmemBytes ? kSlabFullSmemBytes : kSlabSymSmemBytes;
static_assert(kSlabStages % kSlabGroups == 0, "a stage must always return to the same consumer group");
static_assert(kSlabWinBytes % 128 == 0 && kSlabStageBytes % 128 == 0 && kSymStageBytes % 128 == 0,
              "stages must stay 128-byte aligned");
static_assert(kSlabSmemBytes + 2048 <= 232448, "dynamic + static shared memory must fit one block per SM");
static_assert(kSymRows == 2 * kSlabRows, "a symmetric tile is two passes of the group's rows");
static_assert(kSlabRows * kSlabLanesPerRow == 32 * kSlabGroupWarps, "one tile row per lane group");
static_assert(kSlabRowThreads == 32 * kSlabConsumerWarps, "the consumer warps own the rows");
static_assert(kSlabGroups * kSlabRowsPerThread * 16 <= 512, "row records must fit tensor memory");

// A part_info row whose group is {kSlabNoGroup, 0}: the block has no part in that round.
constexpr int kSlabNoGroup = -1;

// Round table of the per-body (batched) launch, rebuilt on the device before every solve
// from the previous solve's per-body iteration counts (pk_pcg_slab.cu,
// slab_schedule_kernel).  Bodies are placed largest estimated work (duration x parts)
// first; a body of k parts takes the k consecutive blocks that are free earliest (ties:
// the lowest first block), all in one round: the round after the latest of those blocks' earlier rounds
// (blocks that reach it sooner idle through the rounds in between, which costs them
// nothing).  Estimated duration of a body: iterations x (c0 + kSlabSchedRowUs x its
// largest part's rows), c0 = kSlabSchedMultiUs for several parts (grid exchanges),
// kSlabSchedSingleUs for one -- per-iteration costs measured on B200; iterations = the
// body's count in the previous solve, or the iteration cap before the first.
constexpr int kSlabSchedThreads = 256;
constexpr int kSlabSchedMaxGrid = 256;
constexpr int kSlabSchedMaxSort = 2048;  // bodies it places (more: the batched layout does not apply)
constexpr float kSlabSchedMultiUs = 8.0f, kSlabSchedSingleUs = 4.0f, kSlabSchedRowUs = 0.012f;

struct SlabScheduleArgs {
    int grid;                  // blocks of the launch (<= kSlabSchedMaxGrid)
    int rounds;                // rounds of the table (>= the number of bodies placed)
    int nbodies;               // bodies with rows
    const int* body_part0;     // [nbodies] first part (plan numbering); a body's parts are consecutive
    const int* body_parts;     // [nbodies] its parts
    const int* plan_info;      // [parts] x kSlabPartInts
    const int* plan_body;      // [parts]
    const BatchBodyStats* body_stats;  // the previous solve's, by body id
    int nstats;                // entries of body_stats
    int max_iterations;
    int* out_info;             // [rounds][grid] x kSlabPartInts
    int* out_body;             // [rounds][grid]
    int* out_rounds;           // [grid]: rounds each block runs
    unsigned* flags;           // kFlagBreakdown when a body finds no room (the host sizes the table)
};

template <class Acc>
struct SlabPcgArgs {
    int n;                       // dynamic rows
    int rounds;                  // parts per block, taken in order (1 for the coupled solve)
    const int* block_rounds;     // [grid]: rounds block b runs (NULL: all)
    const int* part_info;        // [rounds][grid] x kSlabPartInts
    const int4* tile_desc;       // per tile: stream offset / 16, bytes, first local row, rows
    int tile_count;
    int halo_count;
    const unsigned char* stream;
    unsigned long long stream_bytes;
    const int* halo_src;         // slab index of each halo row
    const unsigned char* exported;  // per slab row: 1 when another part's window holds it
    const int* perm;             // slab index -> dynamic row
    const float* b;              // per dynamic row
    const float* minv;
    float* x;                    // per dynamic row: delta-v out
    float* qs;                   // 4 per slab row: q of phase A
    float* ss;                   // 4 per slab row: s published for the window passes
    ExSlot* slots;               // [rounds][2][grid]
    unsigned* group_count;       // [rounds][grid]: arrival counter of the group starting at each block (zeroed)
    GridSync* sync;              // err flag
    int max_iterations;
    Acc tolerance;
    int skip_on_flags;
    int integrate;
    float dt;
    const int* dyn_to_node;
    float* node_x;
    float* node_v;
    unsigned* flags;
    DevStats* stats;
    // Per-body solves (grouped): each block's body, the per-body statistics and the success
    // flags some body lacks; 0 / NULL for the coupled solve (one group of all blocks).
    int grouped;
    const int* part_body;        // [rounds][grid]
    int nbodies;
    BatchBodyStats* body_stats;
    unsigned* missing;
    // Stream form (pk_slab_plan.h): 0 full symmetric rows, 1 the symmetric form (each
    // in-sub-part block once, transposed products through the groups' shared-memory rings).
    int sym;
};

// Polls of one wait of the part-resident and resident kernels for another block: seconds.
constexpr unsigned kTagSpinLimit = 1u << 22;

// ------------------------------------------------------------------ part-resident PCG, coupled
// pk_pcg_part.cu: the window, a ring of as many stages as fit, the table.
constexpr size_t kPartSmemLimit = 224 * 1024;
// Six: with nine the exchange's packets wait behind a longer refill (17.9 against 17.6 us an
// iteration with 122,400 FP32 rows).
constexpr int kPartMaxStages = 6;
constexpr size_t part_stage(size_t real) { return real == 8 ? kWideStageBytes : kSlabStageBytes; }
constexpr size_t part_table(size_t real) { return 16 * size_t(real == 8 ? kWideMaxTiles : kSlabMaxTiles); }
constexpr size_t part_ring_offset(size_t real, int window) { return (3 * real * window + 127) / 128 * 128; }
constexpr int part_stages(size_t real, int window)
{
    const size_t fixed = part_ring_offset(real, window) + part_table(real);
    const size_t fit = fixed < kPartSmemLimit ? (kPartSmemLimit - fixed) / part_stage(real) : 0;
    return fit < size_t(kPartMaxStages) ? int(fit) : kPartMaxStages;
}
static_assert(part_stages(8, kSlabWinCap) >= 4, "the largest window must leave a ring");
template <class Real>
struct PartPcgArgs {
    int n;                       // dynamic rows
    const int* part_info;        // [grid] x kSlabPartInts
    const int* send_start;       // [grid + 1]
    const int2* send;            // {row of the part, halo row}
    const int4* tile_desc;
    int tile_count, halo_count;
    const unsigned char* stream;
    unsigned long long stream_bytes;
    int stages, win_cap;
    unsigned ring_offset;
    unsigned spin_limit;         // polls of one wait for another block
    unsigned char* rows_in;      // a packet (FP64: two) per halo row; zero at launch
    unsigned char* sums_in;      // the blocks' inboxes; zero at launch
    const int* perm;             // slab index -> dynamic row
    const Real* b;             // per dynamic row
    const Real* minv;
    Real* x;                   // per dynamic row: delta-v out
    Real* qs;                  // 4 per slab row
    Real* mrow;                // FP64: M^-1 in slab order, [9][n]
    int float_sums;            // FP32 systems: the sums (in double) are judged as floats
    int max_iterations;
    double tolerance;
    int skip_on_flags, integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
    unsigned* flags;
    DevStats* stats;
};
struct WideFillArgs {
    const double* values;        // the assembled blocks
    int nnz;
    const int4* tile_desc;
    const int* tile_entry0;
    int tile_count, entries;
    const unsigned* fill_src;
    const unsigned char* layout; // headers and columns (SlabPlan::stream): written instead of the blocks
    unsigned char* stream;
    unsigned long long stream_bytes;
};

// ------------------------------------------------------------------ resident PCG
// The resident PCG kernel (pk_pcg_res.cu; layout in pk_res_plan.h): one block per part,
// the part's rows on chip for the whole solve, one exchange per iteration.
template <class Real>
struct ResPcgArgs {
    int n;
    int lpr;                         // lanes per row: 1, 2, 4 or 8
    int nslots;                      // slots per thread
    int tmem_slots;                  // of them in tensor memory
    int max_halo;                    // most halo rows of a part (clusters: the inbox's rows)
    const int* part_info;            // [grid] x kResPartInts
    const int* perm;                 // part order -> dynamic row
    const int* halo_src;
    int halo_count;
    const int2* send;                // rows to send {row of the part, place}, part by part
    const unsigned* src;             // [part's slots][thread]
    const unsigned short* col;
    int slot_count;
    int nnz;
    unsigned smem_bytes;             // dynamic shared memory of the launch
    const Real* values;              // the assembled system
    const Real* b;
    const Real* minv;
    Real* x;                         // per dynamic row: delta-v out
    // exchange through global memory (not in clusters)
    unsigned char* rows_in;          // [2][halo_count] tagged q rows (16 bytes each; 32 in FP64)
    unsigned char* sums_in;          // [2][grid][sender] x kResSlotBytes: tagged sums
    size_t sums_stride;              // bytes of one block's inbox: the largest group's senders
    unsigned* epoch;                 // [grid] tag base of the group starting at each block
    unsigned spin_limit;             // polls of one wait for another block
    int float_sums;                  // FP32 systems: the sums (in double) are judged as floats
    int max_iterations;
    double tolerance;
    int skip_on_flags;
    int integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
    unsigned* flags;
    DevStats* stats;
    // per-body solves (see SlabPcgArgs)
    int grouped;
    int nbodies;
    BatchBodyStats* body_stats;
    unsigned* missing;
};
constexpr int kResSlotBytes = 64;    // four 16-byte packets

// ------------------------------------------------------------------ FP64 refinement
// Kernels of the outer true-residual refinement (pk_refine.cu).
constexpr int kRefineThreads = 256;

template <class Real>
struct RefineArgs {
    BsrView<Real> a;
    const Real* b;           // assembled right-hand side (kept while corrections run)
    const Real* minv;
    const double* x64;       // FP64 solution so far (NULL: x = 0)
    Real* rhs_out;           // residual rounded to Real: the next correction's rhs (may be NULL)
    double* partials;        // 2 per block: r^T M^-1 r, r.r
    int* bad;                // non-finite residual / update flags (cleared by the caller)
    // update
    Real* dx;                // delta-v in the storage type (written by the update)
    int integrate;
    Real dt;
    const int* dyn_to_node;
    Real* node_x;
    Real* node_v;
};

template <class Real>
int refine_residual_blocks(int n);
template <class Real>
cudaError_t launch_refine_residual(const RefineArgs<Real>& args, cudaStream_t stream);
template <class Real>
cudaError_t launch_refine_accumulate(double* x64, const Real* dx, int count, int first, cudaStream_t stream);
// Check pass (delta-v rounded and written to args.dx, finiteness into *args.bad), then, if
// args.integrate, the update of velocities and positions when nothing failed.
template <class Real>
cudaError_t launch_refine_update(const RefineArgs<Real>& args, cudaStream_t stream);

// The FP64 true residual of an FP32-stored step, from the tet data rather than the stored
// blocks: r = b - A x with b = dt f - dt^2 K v + dt m g and A = M + dt^2 K evaluated
// element by element in FP64 (FP64 rest data, FP64 polar rotation and stress), i.e.
//   r_a = sum over a's tets of -(dt S + dt^2 Q(v + x~)) g_a - dt c v_a + dt m g - m x_a
// (Q the folded stiffness, x~ the solution on the dynamic nodes and 0 elsewhere).
template <class Real>
struct ElemResidualArgs {
    int n;                          // dynamic rows
    int node_count;
    int tet_count;
    const int4* tet_nodes;
    const unsigned char* enabled;   // bit 0 simulated, bit 1 linear
    const double* dm_inv;           // FP64 rest data: 9 per tet
    const double* params;           // 4 per tet: rest volume, lambda, mu, damping
    const double* mass;             // FP64, per world node
    const Real* x;                  // node state (storage type)
    const Real* v;
    const int* node_to_dyn;
    const int* dyn_to_node;
    const int* inc_start;
    const int* inc_list;
    const Real* minv;               // block-Jacobi inverse (storage type), for r^T M^-1 r
    const double* x64;              // the FP64 solution so far (NULL: 0)
    double* vx;                     // scratch: per world node v + x~
    double* u;                      // scratch: per tet -(dt S + dt^2 Q(v + x~)), NaN when skipped
    double dt;
    double gravity[3];
    int linear;
    Real* rhs_out;                  // residual rounded to Real (may be NULL)
    double* partials;               // 2 per block: r^T M^-1 r, r.r
    int* bad;
};
template <class Real>
int elem_residual_blocks(int n);
template <class Real>
cudaError_t launch_elem_residual(const ElemResidualArgs<Real>& args, cudaStream_t stream);

// ------------------------------------------------------------------ adjoint step
// Backward element kernel (pk_adjoint.cu): per tet, the sensitivities of
// J = dt w.f(x) - dt^2 w.K(x) z to the tet's node positions (12 doubles) and to its
// log Young's modulus.
template <class Real>
struct AdjointArgs {
    int rows;                // dynamic rows
    int tet_count;
    const int4* nodes;
    const unsigned char* enabled;
    const Real* dm_inv;
    const Real* params;      // V, lambda, mu, damping
    const Real* x;           // per world node
    const Real* v;
    const int* node_to_dyn;
    const int* dyn_to_node;
    const int* inc_start;    // incidence of the dynamic rows, as in AssemblyArgs
    const int* inc_list;
    const double* mass;      // per node
    const double* damping;   // per tet
    double* w;               // adjoint solution, per dynamic row
    double* du;              // the step's delta-v, per dynamic row
    double* g;               // adjoint right-hand side, per dynamic row
    double* xbar;            // per node: the adjoints after the step, then before it
    double* vbar;
    Real* rhs;               // out: g in the storage type
    const Real* solution;    // per dynamic row: of the last solve
    const Real* product;     // A w
    double dt, dt_exact;     // the step's dt in the storage type, and as given
    int linear;
    unsigned* flags;
    double* tet_grad;        // out: 12 per tet
    double* tet_theta;       // out: 1 per tet
};

// Launchers (pk_kernels.cu).  All asynchronous on `stream`.
template <class Real>
cudaError_t launch_tet_kernel(const AssemblyArgs<Real>& args, bool fp64_polar_fallback, cudaStream_t stream);
// Coupled part-resident PCG (pk_pcg_part.cu), cooperative, a block per part.
template <class Real>
int pcg_part_max_grid();
template <class Real>
cudaError_t launch_pcg_part_kernel(const PartPcgArgs<Real>& args, int grid, cudaStream_t stream);
cudaError_t launch_wide_fill_kernel(const WideFillArgs& args, cudaStream_t stream);
// TetView::rest, when the tets are set.
template <class Real>
cudaError_t launch_tet_pack(const Real* dm_inv, const Real* params, Real* rest, int tet_count, cudaStream_t stream);
template <class Real>
cudaError_t launch_visual_kernel(int kind, const int* nodes, const float* weights, const unsigned char* live, int count,
                                 const Real* x, float* verts, float* normals, cudaStream_t stream);
template <class Real>
cudaError_t launch_sphere_contacts(const int* nodes, const unsigned char* flags, const Real* x, int tet_count,
                                   const Real* center, Real radius, int max_out, int* count, int* out_tet,
                                   Real* out_point, cudaStream_t stream);
// Per point connection, before the row kernel: its weighted point and velocity, whether it
// applies this step, and its force (args.conn_eval).
template <class Real>
cudaError_t launch_conn_kernel(const AssemblyArgs<Real>& args, cudaStream_t stream);
template <class Real>
cudaError_t launch_row_kernel(const AssemblyArgs<Real>& args, int max_row_blocks, cudaStream_t stream);
// Builds AssemblyArgs::blk_range and blk_list (4 entries per incidence) for the pattern, the
// incidences and the tets' nodes; counts into *missing (zeroed).
cudaError_t launch_block_list_kernel(int n, const int* row_start, const int* col, const int* inc_start,
                                     const int* inc_list, const int4* tet_nodes, const int* node_to_dyn, int2* range,
                                     unsigned* list, int* missing, cudaStream_t stream);
template <class Real, class Acc>
cudaError_t launch_pcg_kernel(const PcgArgs<Real, Acc>& args, int grid, int threads, cudaStream_t stream);
// Largest cooperative grid (one wave) for the staged (args.ntiles > 0) or unstaged kernel.
template <class Real, class Acc>
int pcg_max_grid(int threads, bool staged);
template <class Real>
cudaError_t launch_spmv_kernel(const BsrView<Real>& a, const Real* x, Real* y, cudaStream_t stream);
// g = vbar + dt xbar on the dynamic rows (into g and rhs); du = the last solution.
template <class Real>
cudaError_t launch_adjoint_rhs_kernel(const AdjointArgs<Real>& args, cudaStream_t stream);
// w = the last solution, in double.
template <class Real>
cudaError_t launch_adjoint_widen_kernel(const AdjointArgs<Real>& args, cudaStream_t stream);
// The nodes' adjoints before the step, from the tets' gradients, in place.
template <class Real>
cudaError_t launch_adjoint_node_kernel(const AdjointArgs<Real>& args, cudaStream_t stream);
template <class Real>
cudaError_t launch_adjoint_tet_kernel(const AdjointArgs<Real>& args, cudaStream_t stream);
// Batched per-body PCG (pk_pcg_batch.cu): cooperative, one block per body part.
template <class Real, class Acc>
cudaError_t launch_pcg_batch_kernel(const BatchPcgArgs<Real, Acc>& args, int grid, cudaStream_t stream);
template <class Real, class Acc>
int pcg_batch_max_grid();
// Ring-staged PCG (pk_pcg_ring.cu): one block of kRingThreads per SM.
template <class Real, class Acc>
cudaError_t launch_pcg_ring_kernel(const RingPcgArgs<Real, Acc>& args, int grid, cudaStream_t stream);
template <class Real, class Acc>
int pcg_ring_max_grid();

// Part-resident PCG (pk_pcg_slab.cu): cooperative, one block of kSlabThreads per part.
template <class Acc>
cudaError_t launch_pcg_slab_kernel(const SlabPcgArgs<Acc>& args, int grid, cudaStream_t stream);
cudaError_t launch_slab_schedule_kernel(const SlabScheduleArgs& args, cudaStream_t stream);
template <class Acc>
int pcg_slab_max_grid();
// Writes the assembled upper blocks and their transposes into the slab stream, tile by
// tile (tile_desc: 4 ints per tile; tile_entry0: ntiles + 1 offsets into fill_src).
cudaError_t launch_slab_fill_kernel(const float* values, int nnz, const int* tile_desc, const int* tile_entry0,
                                    int ntiles, const unsigned* fill_src, int nentries, float* stream,
                                    unsigned long long stream_floats, int sym, cudaStream_t stream_);

// Resident PCG (pk_pcg_res.cu): `grid` blocks of `threads`, in clusters of `cluster` blocks
// or, with 0, as a cooperative launch.
template <class Real>
cudaError_t launch_pcg_res_kernel(const ResPcgArgs<Real>& args, int threads, int rpt, int cluster, int grid,
                                  cudaStream_t stream);
template <class Real>
ResLimits pcg_res_limits();

constexpr int kPcgThreads = 512;

}  // namespace pk
