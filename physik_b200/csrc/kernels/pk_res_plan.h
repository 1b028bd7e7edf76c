// pk_res_plan.h -- host-side layout of the resident PCG kernel (pk_pcg_res.cu).
//
// Where the whole matrix fits the SMs' on-chip memory, a solve needs no matrix traffic at
// all: every block of the launch loads its part's rows once and keeps them in shared memory
// and registers for all iterations.  The layout names what each thread loads and what it
// multiplies it with.
//
// Rows are cut into parts, one per block, by coordinate bisection (per body for per-body
// solves; a body's parts are consecutive blocks: a group).  `lpr` lanes share a row, one
// pass of the block covers the part.  The full symmetric row (upper blocks and transposes
// of the lower ones, by ascending window column) is dealt round-robin to the row's lanes:
// lane l holds entries l, l + lpr, ...  A part of more rows than a block has threads to
// spare gives a thread two rows, t and t + threads, whose entries alternate in its slots.
// Slots live in registers first, then in tensor memory where the launch uses it, then in
// shared memory.  A slot is one entry per thread: src[slot][thread]
// the canonical upper block (kSlabLowerBit: its transpose; kSlabNoPos: none, a zero block)
// and col[slot][thread] three times the window index of its column.
//
// A part's window is its rows, then its halo (the rows of other parts they couple to).
//
// A launch exchanges in one of two ways.  Groups of at most kResMaxCluster blocks run as
// thread-block clusters of `cluster` blocks (a group never straddles two; blocks a cluster
// has left over have no part) and write into each other's shared memory; such a launch may
// have more clusters than fit the GPU at once, since clusters do not wait for each other
// (the runtime asks for a layout only where the whole matrix is within the SMs' memory).
// Larger groups exchange through global memory and must all be resident (cluster = 0, a
// cooperative launch).
// Plain C++ (no CUDA), shared by the runtime and its CPU self-check.
#pragma once

#include <cstddef>
#include <string>
#include <vector>

namespace pk {

constexpr int kResMaxThreads = 512, kResMinThreads = 128;
constexpr int kResPairThreads = 320;  // threads of a block with two rows a thread
// Halo rows a thread takes: compact parts of 600 rows have 450 to 750 (a third row costs 5 %).
constexpr int res_halo_per_thread(int rpt) { return rpt > 1 ? 3 : 2; }
constexpr int kResMaxParts = 160;   // blocks of a group exchanging through global memory
constexpr int kResSlotPoll = kResMaxParts / 32;
constexpr int kResMaxCluster = 16;
// Per part: row0, rows, halo0, halo rows, slot0, (unused), first block and size of its group
// (size 0: the block has no part), body, first and number of its sends.
constexpr int kResPartInts = 12;
constexpr size_t kResAloneBytes = 116 * 1024;  // more than half an SM's: no second block beside this one
constexpr size_t kResSmemLimit = 224 * 1024;  // dynamic shared memory of one block per SM

// Slots that stay in registers: what the register file leaves beside the rows' vectors at
// 128 registers a thread (512 threads), 168 (two rows a thread) or 255 (up to 256 threads).
constexpr int res_reg_slots(int real, int threads, int rpt)
{
    if (rpt > 1) return 2;
    return threads <= 256 ? (real == 4 ? 8 : 4) : (real == 4 ? 4 : 0);
}
// Tensor memory: 512 columns of one word for the warps of a quarter of the lanes (every
// fourth warp), read in batches of 36 words a thread: four FP32 slots or two FP64 slots.
constexpr int kResTmemWords = 36;
constexpr int res_tmem_batch(int real) { return kResTmemWords / (9 * real / 4); }
constexpr int res_tmem_columns(int threads) { return 512 / ((threads / 32 + 3) / 4); }
constexpr int res_tmem_slots(int real, int threads)
{
    return res_tmem_columns(threads) / kResTmemWords * res_tmem_batch(real);
}
constexpr size_t res_align(size_t v) { return (v + 15) & ~(size_t)15; }
constexpr size_t res_row_packet(int real) { return real == 4 ? 16 : 32; }

// Bytes of dynamic shared memory of a part: inbox (clusters: two buffers of sums and of the
// launch's most halo rows), window, halo r and M^-1, q, values of in_smem slots, columns of those
// and of the tensor memory's.
constexpr size_t res_smem_bytes(int real, int threads, int m, int h, int in_smem, int tmem, int cluster,
                                int max_halo)
{
    const size_t inbox = cluster > 0 ? 2 * (size_t)kResMaxCluster * 64 + 2 * (size_t)max_halo * res_row_packet(real) : 0;
    return inbox + res_align(3 * (size_t)(m + h) * real) + res_align(12 * (size_t)h * real) +
           res_align(3 * (size_t)m * real) + res_align((size_t)in_smem * threads * 9 * real) +
           res_align((size_t)(in_smem + tmem) * threads * 2);
}

struct ResPlan {
    int n = 0, parts = 0;         // parts: blocks of the launch, those without rows included
    int lpr = 4, threads = 128, slots = 0, cluster = 0;
    int rpt = 1;                  // rows per thread: 1 (lpr lanes a row) or 2 (one lane a row)
    int tmem = 0;                 // slots in tensor memory, after those in registers
    int smem_slots() const
    {
        const int rest = slots - tmem - res_reg_slots(real, threads, rpt);
        return rest > 0 ? rest : 0;
    }
    int real = 4;
    std::vector<int> perm;        // part order -> dynamic row
    std::vector<int> part_info;   // kResPartInts per part
    std::vector<int> halo_src;    // part-order index of every halo row, part by part
    // What each part sends, part by part: {row of the part, place}, the place the index in
    // halo_src or, in a cluster, (block of the cluster << 16) | halo row of that block.
    std::vector<int> send;
    int max_group = 1, max_halo = 0, max_rows = 0;
    std::vector<unsigned> src;    // [part's slots][thread]
    std::vector<unsigned short> col;
    size_t smem_bytes = 0;        // most of any part
};

// What the GPU holds: blocks of a cooperative launch, and clusters of 1, 2, 4, 8, 16 blocks
// resident at once (0: not available).
struct ResLimits {
    int blocks = 0;
    int clusters[5] = {0, 0, 0, 0, 0};
};

// Builds the layout for the bodies (segments [seg[b], seg[b + 1]), covering all rows; no
// block couples two of them), real = sizeof(Real).  coords: 3 doubles per row.  Returns ""
// on success, otherwise why it does not apply (more than on-chip memory holds); `out` is
// then unusable.
std::string build_res_plan(int n, const int* row_start, const int* col, const int* lt_start, const int* lt_row,
                           const int* lt_block, const double* coords, const int* seg, int nseg,
                           const ResLimits& limits, int real, ResPlan& out);

// The conditions the kernel checks before it uses a part, and that every block is placed
// once (its transpose once, off the diagonal) and every halo row's owner sends it, in the
// same group.  "" when they hold.
std::string res_check(const ResPlan& plan, int nnz, const ResLimits& limits, int real);

// y = A x through the plan as the kernel's lanes read it, in double (the CPU self-check).
void res_spmv_host(const ResPlan& plan, const double* values, const double* x, double* y);

}  // namespace pk
