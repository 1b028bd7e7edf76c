// pk_pcg_res.cu -- the resident cooperative block-Jacobi PCG kernel.
//
// The solve of the other PCG kernels (SolvePreconditionedConjugateGradient,
// src/Core/Solvers/Linear/ConjugateGradientSolver.cpp:114-241, with the SpMV of
// SparseBlockMatrix::Multiply, src/Math/SparseBlockMatrix.cpp:209-268, and
// World::IntegrateImplicitEuler, src/Core/World/World.cpp:644-695, fused at the end) for
// systems whose matrix fits the SMs' on-chip memory (pk_res_plan.h).  Such a solve is bound
// by latency, not by bytes: an iteration of the streaming kernels spends most of its time
// in two grid exchanges and the loads around them.  Here
//
// * every block loads its part's rows once, straight from the assembled blocks, into
//   registers, tensor memory and shared memory; x, r, s, d and M^-1 of a row stay in the
//   registers of the lane that owns it.
// * parts of more than 256 rows (FP32) give a thread two rows and keep most of the blocks in
//   tensor memory: a warp's tcgen05.ld of 36 words a thread brings four blocks without using
//   the shared memory's bandwidth, and its 256 KB beside the 224 KB of shared memory hold a
//   part of 640 rows of 15 blocks (94,000 rows on the GPU).  FP64 uses it where registers and
//   shared memory are too small.
// * an iteration has one exchange.  The blocks publish, with the partial sums of d.q, the
//   rows of q = A d that other parts' windows hold; every block then knows alpha and beta
//   and updates r, s = M^-1 r and d of its halo rows itself, with the same operations as
//   their owners (so all copies of a row agree bit for bit).  beta needs r'.s' of the
//   updated vectors before they exist; it is predicted from sums of the same exchange,
//       r'.s' = r.s - alpha (q.s + r.z) + alpha^2 q.z,   z = M^-1 q, r' = r - alpha q
//   (exact in exact arithmetic for any M), and the true r'.s' of the updated vectors is
//   summed with the next exchange and used for alpha, for the stopping test and for the
//   next prediction ("predict and recompute", Chen and Carson 2020).  Where the prediction
//   would cancel (r'.s' below a sixteenth of r.s), near the stopping target and in the last
//   iteration the true sum is exchanged at once.
// * through global memory an exchange needs no fence: every value travels in a 16-byte packet with a tag (the
//   exchange's number), written and read whole.  A sender writes into the inbox of every
//   reader, so that a reader polls lines nobody else reads, and reads them coalesced.  Two
//   buffers by parity: a block overwrites exchange g's packets in g + 2, after it has seen
//   every block's sums of g + 1, which a block sends only when it has read all of g.  Tags
//   go on from solve to solve (epoch), so nothing is cleared between solves.
//
// Measured per CG iteration against the streaming kernels (part-resident stream for FP32
// storage, ring for FP64): 8x8x8 box FP32 2.3 us (7.2), 32x8x8 beam FP64 3.0 us (13.3),
// 64x16x16 beam 3.5 us mixed (10.9) and 4.3 us FP64 (18.5), 61x47x29 block mixed (594 rows a
// part) 7.0 us (19.3).  What is left is a chain of
// latencies: about 3,000 cycles of a block's own work (product, two sets of FP64 sums by
// shuffles, the scalars, the updates; 8.6 cycles an FP64 add, 24 a shuffle, 45 a barrier of
// 512 threads) and the exchange.
//
// All sums keep one fixed order: warp shuffles, then the block's warps, then the group's
// blocks, the same in every block; a run repeats bit for bit.  Sums and scalars are FP64 in
// every precision (an FP32 system's sums are judged as floats).  Every wait is bounded; one that gives up sets the timeout flag, which
// ends the other blocks' waits.
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "pk_device.cuh"
#include "pk_exchange.cuh"

namespace pk {
namespace {

constexpr int kResMaxWarps = kResMaxThreads / 32;
constexpr int kResSums = 4;  // d.q, q.s + r.z, q.z, r.s; at the end r.r in the first
constexpr int kResSendRegs = 2;

// ------------------------------------------------------------------ cluster exchange
__device__ __forceinline__ unsigned cluster_map(const void* p, unsigned rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async16(unsigned dst, Packet v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(v.lo), "l"(v.hi), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async8(unsigned dst, unsigned long long v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(v),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async_row(unsigned dst, V3<float> q, unsigned bar)
{
    st_async16(dst, {(unsigned long long)__float_as_uint(q.x) | ((unsigned long long)__float_as_uint(q.y) << 32),
                     (unsigned long long)__float_as_uint(q.z)},
               bar);
}
__device__ __forceinline__ void st_async_row(unsigned dst, V3<double> q, unsigned bar)
{
    st_async16(dst, {(unsigned long long)__double_as_longlong(q.x), (unsigned long long)__double_as_longlong(q.y)}, bar);
    st_async8(dst + 16, (unsigned long long)__double_as_longlong(q.z), bar);
}
template <class Real>
constexpr unsigned row_tx_bytes()
{
    return sizeof(Real) == 4 ? 16 : 24;
}
// Bounded wait for the phase with the given parity, seeing what cluster peers wrote.
__device__ __forceinline__ bool cluster_wait(unsigned long long* bar, unsigned parity, unsigned limit)
{
    for (unsigned i = 0; i < limit; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 36 words of a thread's tensor memory (the warp's lanes, 36 columns), each waiting for its
// own completion.
struct Words {
    unsigned w[kResTmemWords];
};
#define PK_W(i) "=r"(t.w[i]), "=r"(t.w[i + 1]), "=r"(t.w[i + 2]), "=r"(t.w[i + 3])
__device__ __forceinline__ void tmem_ld36(unsigned addr, Words& t)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%36];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%32,%33,%34,%35}, [%37];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : PK_W(0), PK_W(4), PK_W(8), PK_W(12), PK_W(16), PK_W(20), PK_W(24), PK_W(28), PK_W(32)
        : "r"(addr), "r"(addr + 32u)
        : "memory");
}
#undef PK_W
#define PK_W(i) "r"(t.w[i]), "r"(t.w[i + 1]), "r"(t.w[i + 2]), "r"(t.w[i + 3])
__device__ __forceinline__ void tmem_st36(unsigned addr, const Words& t)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%36], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
        "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};\n\t"
        "tcgen05.st.sync.aligned.32x32b.x4.b32 [%37], {%32,%33,%34,%35};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::PK_W(0),
        PK_W(4), PK_W(8), PK_W(12), PK_W(16), PK_W(20), PK_W(24), PK_W(28), PK_W(32), "r"(addr), "r"(addr + 32u)
        : "memory");
}
#undef PK_W
__device__ __forceinline__ float words_at(const Words& t, int i, float) { return __uint_as_float(t.w[i]); }
__device__ __forceinline__ double words_at(const Words& t, int i, double)
{
    return __hiloint2double((int)t.w[2 * i + 1], (int)t.w[2 * i]);
}
__device__ __forceinline__ void words_set(Words& t, int i, float v) { t.w[i] = __float_as_uint(v); }
__device__ __forceinline__ void words_set(Words& t, int i, double v)
{
    t.w[2 * i] = (unsigned)__double2loint(v);
    t.w[2 * i + 1] = (unsigned)__double2hiint(v);
}

// MAXT: threads per block at most (256 leaves a thread twice the registers of 512).
// CL: exchange inside a cluster (else through global memory).
// R: rows per thread (2: one lane a row, rows tid and tid + T, whose entries alternate in the
// slots).  TM: slots in tensor memory.  FS: the sums judged as floats (as_float_sum; a run-time
// rule cost every precision 1.5 % of an iteration, these instances cost FP32 alone).
template <class Real, int MAXT, bool CL, int R, bool TM, bool FS>
__global__ void __launch_bounds__(MAXT, 1) pcg_res_kernel(ResPcgArgs<Real> P)
{
    constexpr int KR = res_reg_slots(sizeof(Real), MAXT, R);
    constexpr int KB = res_tmem_batch(sizeof(Real));
    static_assert(KR % R == 0 && KB % R == 0, "a slot's row is known at compile time");
    constexpr int NH = res_halo_per_thread(R);
    constexpr int RB = (int)res_row_packet(sizeof(Real));
    extern __shared__ __align__(128) unsigned char dyn[];
    // the owner warps' partials and the group's sums, by exchange parity
    __shared__ double sh_part[2][kResSums * kResMaxWarps];
    __shared__ double sh_sum[2][kResSums];
    __shared__ unsigned sh_bits[3], sh_gbits[3];  // flags by exchange number
    __shared__ __align__(8) unsigned long long sh_bar[2];
    __shared__ int s_fail;
    __shared__ unsigned s_tmem;

    const int T = blockDim.x, W = T >> 5, lpr = P.lpr;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x;
    const int* pi = P.part_info + (size_t)kResPartInts * blk;
    const int row0 = __ldg(pi + 0), halo0 = __ldg(pi + 2), slot0 = __ldg(pi + 4), body = __ldg(pi + 8),
              send0 = __ldg(pi + 9);
    int m = __ldg(pi + 1), h = __ldg(pi + 3), gfirst = __ldg(pi + 6), gsize = __ldg(pi + 7), sends_n = __ldg(pi + 10);
    const unsigned in_flags = *(volatile unsigned*)P.flags;
    const bool skip = P.skip_on_flags && (in_flags & (kFlagPrecomputeFailed | kFlagSingularDiag));
    const bool idle = CL && gsize == 0;  // a block its cluster has left over
    unsigned cl_size = 1;
    if (CL) asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cl_size));
    const int cl0 = CL ? blk - blk % (int)cl_size : 0;
    unsigned bad0 = 0;
    // A part that does not fit the launch (the host never builds one) is emptied and
    // reports a breakdown; a block outside its group works alone.
    if (!idle &&
        (gfirst < 0 || gsize < 1 || gsize > (CL ? kResMaxCluster : kResMaxParts) || gfirst + gsize > (int)gridDim.x ||
         blk < gfirst || blk >= gfirst + gsize || (P.grouped && (unsigned)body >= (unsigned)P.nbodies) ||
         (!P.grouped && (gfirst != 0 || (!CL && gsize != (int)gridDim.x))) ||
         (CL && (gfirst < cl0 || gfirst + gsize > cl0 + (int)cl_size)))) {
        gfirst = blk;
        gsize = 1;
        bad0 = 4u;
    }
    int nslots = P.nslots;
    // (the launch's tensor memory: the host's rule, else none)
    const int tslots = TM && P.tmem_slots > 0 && P.tmem_slots <= res_tmem_slots(sizeof(Real), T) &&
                               P.tmem_slots % KB == 0 && P.smem_bytes >= kResAloneBytes
                           ? P.tmem_slots
                           : 0;
    const int s0 = KR + tslots;  // first slot in shared memory
    if (m < 0 || m * lpr > T * R || (R > 1 && lpr != 1) || nslots % R != 0 || h < 0 || h > NH * T || h > P.max_halo ||
        row0 < 0 || row0 + m > P.n || halo0 < 0 || halo0 + h > P.halo_count || sends_n < 0 || send0 < 0 ||
        send0 + sends_n > P.halo_count || nslots < 0 || slot0 < 0 || slot0 + nslots > P.slot_count ||
        res_smem_bytes(sizeof(Real), T, m, h, max(0, nslots - s0), tslots, CL ? 1 : 0, P.max_halo) > P.smem_bytes) {
        m = h = nslots = sends_n = 0;
        bad0 = 4u;
    }
    const bool leader = !idle && blk == gfirst;
    BatchBodyStats* const bs = P.grouped ? P.body_stats + ((unsigned)body < (unsigned)P.nbodies ? body : 0) : nullptr;
    if (skip) {
        if (leader && tid == 0) {
            if (P.grouped) {
                bs->iterations = 0;
                bs->converged = 0;
                bs->residual_norm = 0.0;
                bs->flags = 0;
            } else {
                P.stats->iterations = 0;
                P.stats->converged = 0;
                P.stats->residual_norm = 0.0;
            }
        }
        return;
    }
    // Inboxes of a cluster (at the same place in every block): sums [parity][sender][sum],
    // halo rows [parity][row].
    unsigned char* const sums_in = dyn;
    unsigned char* const rows_in = dyn + 2 * kResMaxCluster * kResSlotBytes;
    size_t off = CL ? 2 * (size_t)kResMaxCluster * kResSlotBytes + 2 * (size_t)P.max_halo * RB : 0;
    const int wn = m + h;
    Real* const win = reinterpret_cast<Real*>(dyn + off);
    off += res_align(3 * (size_t)wn * sizeof(Real));
    Real* const hr = reinterpret_cast<Real*>(dyn + off);  // halo r: [3][h], then M^-1: [9][h]
    Real* const hm = hr + 3 * (size_t)h;
    off += res_align(12 * (size_t)h * sizeof(Real));
    Real* const qbuf = reinterpret_cast<Real*>(dyn + off);  // q of the part's rows
    off += res_align(3 * (size_t)m * sizeof(Real));
    // [slot][thread][element]: nine words apart, so a warp's reads hit different banks
    Real* const vals = reinterpret_cast<Real*>(dyn + off);
    off += res_align((size_t)max(0, nslots - s0) * T * 9 * sizeof(Real));
    unsigned short* const cols = reinterpret_cast<unsigned short*>(dyn + off);
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) sh_bits[i] = sh_gbits[i] = 0u;
        s_fail = 0;
        if (CL) {
            mbar_init(&sh_bar[0], 1);
            mbar_init(&sh_bar[1], 1);
            mbar_fence_init();
        }
    }
    if (TM && tslots > 0 && warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (TM) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    unsigned epoch = 0u;
    if (!CL && gsize > 1) epoch = *(volatile unsigned*)(P.epoch + gfirst);
    if (CL)
        cluster_barrier();  // every block's barriers exist before anybody writes to them
    else
        __syncthreads();
    if (TM) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem0 = TM && tslots > 0 ? s_tmem + ((32u * (unsigned)(warp & 3)) << 16) +
                                                   (unsigned)(warp >> 2) * (unsigned)res_tmem_columns(T)
                                             : 0u;
    if (idle) {
        cluster_barrier();
        return;
    }

    // Thread i owns row i < m (R = 2: and row i + T): its vectors and M^-1 stay in its
    // registers.  Packing the rows into the first warps keeps the FP64 work of the sums off the
    // others.  The last threads hold the halo rows.
    bool has[R];
#pragma unroll
    for (int p = 0; p < R; ++p) has[p] = tid + p * T < m;
    const int owner_warps = ((R == 1 ? m : min(m, T)) + 31) / 32;
    // the row that this thread's lane group completes (R = 1; m: none)
    const int qrow = tid % lpr == 0 ? tid / lpr : m;
    const int htid = T - 1 - tid;
    const V3<Real> zero{Real(0), Real(0), Real(0)};
    int cidx[R];
    // the rows this thread sends {row, place}: the first few in registers
    int2 send[kResSendRegs];
#pragma unroll
    for (int u = 0; u < kResSendRegs; ++u)
        send[u] = tid + u * T < sends_n ? __ldg(P.send + send0 + tid + u * T) : make_int2(-1, -1);
    V3<Real> xv[R], rv[R], sv[R], dv[R], qv[R];
    Real mi[R][9];
    unsigned bad = bad0;
#pragma unroll
    for (int p = 0; p < R; ++p) {
        xv[p] = rv[p] = sv[p] = dv[p] = qv[p] = zero;
        cidx[p] = -1;
#pragma unroll
        for (int e = 0; e < 9; ++e) mi[p][e] = Real(0);
        if (has[p]) {
            const int c = __ldg(P.perm + row0 + tid + p * T);
            if ((unsigned)c >= (unsigned)P.n) {
                bad |= 4u;
            } else {
                cidx[p] = c;
                rv[p] = ld3(P.b, c);
#pragma unroll
                for (int e = 0; e < 9; ++e) mi[p][e] = __ldg(P.minv + 9 * (size_t)c + e);
            }
        }
    }
    // Halo rows: r = b and M^-1 in shared memory, d = s in the window.
#pragma unroll
    for (int u = 0; u < NH; ++u) {
        const int j = htid + u * T;
        if (j < h) {
            const int g = __ldg(P.halo_src + halo0 + j);
            int c = 0;
            if ((unsigned)g < (unsigned)P.n) c = __ldg(P.perm + g);
            if ((unsigned)g >= (unsigned)P.n || (unsigned)c >= (unsigned)P.n) {
                c = 0;
                bad |= 4u;
            }
            const V3<Real> b = ld3(P.b, c);
            Real hmi[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                hmi[e] = __ldg(P.minv + 9 * (size_t)c + e);
                hm[(size_t)e * h + j] = hmi[e];
            }
            hr[j] = b.x;
            hr[h + j] = b.y;
            hr[2 * h + j] = b.z;
            const V3<Real> s = apply_minv(hmi, b);
            Real* d = win + 3 * (m + j);
            d[0] = s.x;
            d[1] = s.y;
            d[2] = s.z;
        }
    }
    // The part's blocks: the first KR slots in registers, then those in tensor memory, the
    // others in shared memory.
    Real rval[KR > 0 ? KR : 1][9];
    int rcol[KR > 0 ? KR : 1];
    auto load_entry = [&](int slot, Real (&v)[9]) -> int {
        const size_t at = (size_t)(slot0 + slot) * T + tid;
        const unsigned s = __ldg(P.src + at);
        const int c = __ldg(P.col + at);
        const unsigned k = s & ~kSlabLowerBit;
        const bool live = s != kSlabNoPos && k < (unsigned)P.nnz;
        const Real* q = P.values + 9 * (size_t)(live ? k : 0u);
        Real t[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) t[e] = live ? __ldg(q + e) : Real(0);
        const bool tr = (s & kSlabLowerBit) != 0u;
#pragma unroll
        for (int e = 0; e < 9; ++e) v[e] = tr ? t[3 * (e % 3) + e / 3] : t[e];
        return c + 2 < 3 * wn ? c : 0;
    };
#pragma unroll
    for (int k = 0; k < KR; ++k) {
        rcol[k] = 0;
#pragma unroll
        for (int e = 0; e < 9; ++e) rval[k][e] = Real(0);
        if (k < nslots) rcol[k] = load_entry(k, rval[k]);
    }
    // (columns of all but the register slots go to shared memory)
    for (int k0 = KR; TM && k0 < s0; k0 += KB) {
        Words t;
#pragma unroll
        for (int u = 0; u < KB; ++u) {
            Real v[9] = {};
            const int c = k0 + u < nslots ? load_entry(k0 + u, v) : 0;
#pragma unroll
            for (int e = 0; e < 9; ++e) words_set(t, 9 * u + e, v[e]);
            cols[(size_t)(k0 + u - KR) * T + tid] = (unsigned short)c;
        }
        __syncwarp();
        tmem_st36(tmem0 + (unsigned)((k0 - KR) / KB * kResTmemWords), t);
    }
#pragma unroll 2
    for (int k = s0; k < nslots; ++k) {
        Real v[9];
        const size_t at = (size_t)(k - s0) * T + tid;
        cols[(size_t)(k - KR) * T + tid] = (unsigned short)load_entry(k, v);
#pragma unroll
        for (int e = 0; e < 9; ++e) vals[9 * at + e] = v[e];
    }

    unsigned fl = 0;
    int iterations = 0, it = 0, node[R];
    bool converged = false, have_x = true, timed_out = false;
    bool ran = false;      // the iteration was entered: the residual norm is reported
    bool pending = false;  // the last iteration's r.s comes with the next exchange
    double residual = 0.0, delta = 0.0, target = 0.0, rs_next = 0.0;
    unsigned sbad = 0, gen = 0;
    V3<Real> hq[NH], hs[NH], nx[R], nv[R];
#pragma unroll
    for (int u = 0; u < NH; ++u) hq[u] = hs[u] = zero;
#pragma unroll
    for (int p = 0; p < R; ++p) {
        node[p] = 0;
        nx[p] = nv[p] = zero;
        if (has[p] && cidx[p] >= 0) {
            if (!finite3(rv[p])) bad |= 1u;
            sv[p] = apply_minv(mi[p], rv[p]);
            bool fin = finite3(sv[p]);
#pragma unroll
            for (int e = 0; e < 9; ++e) fin = fin && isfinite(mi[p][e]);
            if (!fin) bad |= 2u;
            dv[p] = sv[p];
            rs_next += dot_acc<double>(rv[p], sv[p]);
        }
        if (has[p]) {
            Real* d = win + 3 * (tid + p * T);
            d[0] = dv[p].x;
            d[1] = dv[p].y;
            d[2] = dv[p].z;
        }
    }

    // The end of an iteration whose r.s is known: false ends the solve.
    auto close = [&](double new_delta, unsigned broken, int done) -> bool {
        if (broken) {
            fl |= kFlagBreakdown;
            return false;
        }
        const double old = delta;
        delta = new_delta;
        // (the last test: delta / old overflows)
        if (!isfinite(delta) || !isfinite(old) || old <= 0.0 || (old < 1.0 && fabs(delta) > scalar_max<FS>() * old)) {
            fl |= kFlagBreakdown;
            return false;
        }
        iterations = done;
        return true;
    };

    // One exchange per turn, whatever it is for: the first residual, an iteration's
    // products, a true r.s at once, the end.
    enum Turn { kFirst, kProducts, kConfirm, kEnd };
    Turn turn = kFirst;
    for (;;) {
        double v[kResSums] = {0.0, 0.0, 0.0, 0.0};
        unsigned bits = 0;
        if (turn == kProducts) {
            // q = A d for the part's rows.
            V3<Real> acc[R];
#pragma unroll
            for (int p = 0; p < R; ++p) acc[p] = zero;
            auto mul = [&](V3<Real>& y, const auto& e, const Real* d) {
                const Real dx = d[0], dy = d[1], dz = d[2];
                y.x += e(0) * dx + e(3) * dy + e(6) * dz;
                y.y += e(1) * dx + e(4) * dy + e(7) * dz;
                y.z += e(2) * dx + e(5) * dy + e(8) * dz;
            };
            auto mul_regs = [&](auto count) {
#pragma unroll
                for (int k = 0; k < decltype(count)::value; ++k) {
                    const Real* d = win + rcol[k];
                    const Real dx = d[0], dy = d[1], dz = d[2];
                    V3<Real>& y = acc[k % R];
                    y.x += rval[k][0] * dx + rval[k][3] * dy + rval[k][6] * dz;
                    y.y += rval[k][1] * dx + rval[k][4] * dy + rval[k][7] * dz;
                    y.z += rval[k][2] * dx + rval[k][5] * dy + rval[k][8] * dz;
                }
            };
            if (KR > 0) {  // (a slot the plan does not have is a zero block)
                if (nslots > KR / 2)
                    mul_regs(std::integral_constant<int, KR>{});
                else if (nslots > KR / 4)
                    mul_regs(std::integral_constant<int, KR / 2>{});
                else
                    mul_regs(std::integral_constant<int, (KR + 3) / 4>{});
            }
            const unsigned short* cp = cols + tid;
            if (TM) {
                for (int k0 = KR; k0 < s0; k0 += KB, cp += KB * T) {
                    const Real* d[KB];
#pragma unroll
                    for (int u = 0; u < KB; ++u) d[u] = win + cp[u * T];
                    Words t;
                    tmem_ld36(tmem0 + (unsigned)((k0 - KR) / KB * kResTmemWords), t);
#pragma unroll
                    for (int u = 0; u < KB; ++u)
                        mul(acc[u % R], [&](int e) { return words_at(t, 9 * u + e, Real()); }, d[u]);
                }
            }
            if constexpr (R == 1) {
                const Real* e = vals + 9 * tid;
#pragma unroll 4
                for (int k = s0; k < nslots; ++k, cp += T, e += 9 * T) {
                    const Real* d = win + *cp;
                    const Real dx = d[0], dy = d[1], dz = d[2];
                    acc[0].x += e[0] * dx + e[3] * dy + e[6] * dz;
                    acc[0].y += e[1] * dx + e[4] * dy + e[7] * dz;
                    acc[0].z += e[2] * dx + e[5] * dy + e[8] * dz;
                }
            } else {
                const Real* e = vals + 9 * tid;
#pragma unroll 2
                for (int k = s0; k < nslots; k += R)
#pragma unroll
                    for (int p = 0; p < R; ++p, cp += T, e += 9 * T)
                        mul(acc[p], [&](int i) { return e[i]; }, win + *cp);
            }
            if (R == 1) {
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    if (lpr > o) {
                        acc[0].x += __shfl_xor_sync(0xffffffffu, acc[0].x, o);
                        acc[0].y += __shfl_xor_sync(0xffffffffu, acc[0].y, o);
                        acc[0].z += __shfl_xor_sync(0xffffffffu, acc[0].z, o);
                    }
            }
#pragma unroll
            for (int p = 0; p < R; ++p) {
                const int row = R == 1 ? qrow : tid + p * T;
                if (row < m) {
                    Real* q = qbuf + 3 * row;
                    q[0] = acc[p].x;
                    q[1] = acc[p].y;
                    q[2] = acc[p].z;
                }
            }
            __syncthreads();
            bits = sbad;
            // The rows other parts hold, spread over all threads (a corner row has many
            // readers: sent by its owner alone it held the block up by 1,500 cycles).
            auto send_row = [&](int2 s) {
                if ((unsigned)s.x >= (unsigned)m) return;
                const V3<Real> q{qbuf[3 * s.x], qbuf[3 * s.x + 1], qbuf[3 * s.x + 2]};
                if (CL) {
                    const unsigned rank = (unsigned)s.y >> 16, j = (unsigned)s.y & 0xffffu;
                    if (rank < cl_size && j < (unsigned)P.max_halo)
                        st_async_row(cluster_map(rows_in + ((size_t)(it & 1) * P.max_halo + j) * RB, rank), q,
                                     cluster_map(&sh_bar[(gen + 1u) & 1u], rank));
                } else if ((unsigned)s.y < (unsigned)P.halo_count) {
                    st_row(P.rows_in + ((size_t)(it & 1) * P.halo_count + s.y) * RB, q, epoch + gen + 1u);
                }
            };
#pragma unroll
            for (int u = 0; u < kResSendRegs; ++u) send_row(send[u]);
            for (int e = tid + kResSendRegs * T; e < sends_n; e += T) send_row(__ldg(P.send + send0 + e));
#pragma unroll
            for (int p = 0; p < R; ++p)
                if (has[p]) {
                    const Real* q = qbuf + 3 * (tid + p * T);
                    qv[p] = V3<Real>{q[0], q[1], q[2]};
                    if (!finite3(qv[p])) bits |= 1u;
                    const V3<Real> z = apply_minv(mi[p], qv[p]);
                    const double dq = dot_acc<double>(dv[p], qv[p]), qz = dot_acc<double>(qv[p], z),
                                 slope = dot_acc<double>(qv[p], sv[p]) + dot_acc<double>(rv[p], z);
                    v[0] = p == 0 ? dq : v[0] + dq;
                    v[1] = p == 0 ? slope : v[1] + slope;
                    v[2] = p == 0 ? qz : v[2] + qz;
                }
            v[3] = rs_next;
        } else if (turn == kEnd) {
            // delta-v back in dynamic-row order; the solve succeeds when it is present and
            // finite; integration is all-or-nothing.
#pragma unroll
            for (int p = 0; p < R; ++p) {
                if (has[p]) v[0] += dot_acc<double>(rv[p], rv[p]);
                if (has[p] && cidx[p] >= 0) {
                    if (!have_x) xv[p] = zero;
                    st3(P.x, cidx[p], xv[p]);
                    if (!finite3(xv[p])) bits |= 1u;
                    if (P.integrate) {
                        node[p] = __ldg(P.dyn_to_node + cidx[p]);
                        const V3<Real> xo = ldplain3(P.node_x, node[p]), vo = ldplain3(P.node_v, node[p]);
                        nv[p] = vo + xv[p];
                        nx[p] = xo + nv[p] * P.dt;
                        if (!finite3(xo) || !finite3(vo) || !finite3(nv[p]) || !finite3(nx[p])) bits |= 2u;
                    }
                }
            }
        } else {
            v[3] = rs_next;
            bits = turn == kFirst ? bad : sbad;
        }

        // ---- the exchange: the group's sums of v and the OR of bits; with the products,
        // also the halo rows of q (hq)
        {
            const bool rows = turn == kProducts;
            ++gen;
            // The owner warps' four sums, each in one butterfly: two steps that halve the
            // values a lane carries, then (lane >> 3) holds its own sum.
            if (warp < owner_warps) {
                const bool up = (lane & 16) != 0, right = (lane & 8) != 0;
                double k0 = up ? v[2] : v[0], k1 = up ? v[3] : v[1];
                k0 += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
                k1 += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
                double t = right ? k1 : k0;
                t += __shfl_xor_sync(0xffffffffu, right ? k0 : k1, 8);
                t += __shfl_xor_sync(0xffffffffu, t, 4);
                t += __shfl_xor_sync(0xffffffffu, t, 2);
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                if ((lane & 7) == 0) sh_part[gen & 1u][(lane >> 3) * kResMaxWarps + warp] = t;
            }
            if (bits) atomicOr(&sh_bits[gen % 3u], bits);
            if (CL && gsize > 1 && tid == 0)
                mbar_arrive_expect_tx(&sh_bar[gen & 1u], (unsigned)gsize * kResSlotBytes +
                                                             (rows ? (unsigned)h * row_tx_bytes<Real>() : 0u));
            __syncthreads();
            if (tid == 0) sh_bits[(gen + 2u) % 3u] = 0u;
            // The block's sums: lane (k, i) takes the partials of sum k of owner warps i and
            // i + 8, then a butterfly over i as far as there are any.  Warps that send do it
            // each for itself; a group of one block needs nothing else.
            const bool sends = gsize > 1 && 8 * warp < gsize;
            if (gsize == 1 || sends) {
                const double* q = sh_part[gen & 1u] + (lane >> 3) * kResMaxWarps + (lane & 7);
                double t = (lane & 7) < owner_warps ? q[0] : 0.0;
                if (owner_warps > 8) t += (lane & 7) + 8 < owner_warps ? q[8] : 0.0;
                if (owner_warps > 4) t += __shfl_xor_sync(0xffffffffu, t, 4);
                if (owner_warps > 2) t += __shfl_xor_sync(0xffffffffu, t, 2);
                if (owner_warps > 1) t += __shfl_xor_sync(0xffffffffu, t, 1);
                const unsigned w = sh_bits[gen % 3u];
                if (gsize == 1) {
#pragma unroll
                    for (int k = 0; k < kResSums; ++k) v[k] = __shfl_sync(0xffffffffu, t, 8 * k);
                    bits = w;
                } else {
                    // warp w's lane (k, i) sends sum k to the group's blocks 8 w + i, + 8 W, ...
                    t = __shfl_sync(0xffffffffu, t, lane & 24);
                    const unsigned long long lo = (unsigned long long)__double_as_longlong(t);
                    if (CL) {
                        const int d = 8 * warp + (lane & 7);
                        if (d < gsize) {
                            const unsigned rank = (unsigned)(gfirst - cl0 + d);
                            st_async16(cluster_map(sums_in + ((gen & 1u) * kResMaxCluster + (unsigned)(blk - gfirst)) *
                                                                 kResSlotBytes + 16 * (lane >> 3),
                                                   rank),
                                       {lo, (unsigned long long)w}, cluster_map(&sh_bar[gen & 1u], rank));
                        }
                    } else {
                        unsigned char* out = P.sums_in + ((size_t)(gen & 1u) * gridDim.x + gfirst) * P.sums_stride +
                                             (size_t)(blk - gfirst) * kResSlotBytes + 16 * (lane >> 3);
                        for (int d = 8 * warp + (lane & 7); d < gsize; d += 8 * W)
                            st_packet(out + (size_t)d * P.sums_stride,
                                      {lo, (unsigned long long)w | ((unsigned long long)(epoch + gen) << 32)});
                    }
                }
            }
            if (CL && gsize > 1) {
                if (!cluster_wait(&sh_bar[gen & 1u], ((gen - 1u) >> 1) & 1u, P.spin_limit)) s_fail = 1;
                __syncthreads();
                const unsigned char* in = sums_in + (size_t)(gen & 1u) * kResMaxCluster * kResSlotBytes +
                                          16 * (lane >> 3);
                double t = 0.0;
                unsigned w = 0;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int i = (lane & 7) + 8 * j;
                    if (i < gsize) {
                        const Packet pk = *reinterpret_cast<const Packet*>(in + (size_t)i * kResSlotBytes);
                        t += __longlong_as_double((long long)pk.lo);
                        w |= (unsigned)pk.hi;
                    }
                }
                if (gsize > 4) t += __shfl_xor_sync(0xffffffffu, t, 4);
                if (gsize > 2) t += __shfl_xor_sync(0xffffffffu, t, 2);
                t += __shfl_xor_sync(0xffffffffu, t, 1);
#pragma unroll
                for (int k = 0; k < kResSums; ++k) v[k] = __shfl_sync(0xffffffffu, t, 8 * k);
                bits = __reduce_or_sync(0xffffffffu, w);
                if (rows)
#pragma unroll
                    for (int u = 0; u < NH; ++u) {
                        const int j = htid + u * T;
                        if (j < h) {
                            const Real* q =
                                reinterpret_cast<const Real*>(rows_in + ((size_t)(it & 1) * P.max_halo + j) * RB);
                            hq[u] = V3<Real>{q[0], q[1], q[2]};
                        }
                    }
                timed_out = s_fail != 0;
            } else if (gsize > 1) {
                // This block's inbox: four warps each take one sum, lane i of them blocks i,
                // i + 32, ...  With rows, the halo threads take their rows.  All reads of a
                // poll are in flight together.
                const int sum = W >= 8 ? warp - 4 : warp;
                const bool polls = sum >= 0 && sum < kResSums;
                const unsigned tag = epoch + gen;
                const unsigned char* in = P.sums_in + ((size_t)(gen & 1u) * gridDim.x + blk) * P.sums_stride + 16 * sum;
                const unsigned char* qin = P.rows_in + ((size_t)(it & 1) * P.halo_count + halo0) * RB;
                Packet pk[kResSlotPoll];
                unsigned todo = 0;
#pragma unroll
                for (int j = 0; j < kResSlotPoll; ++j) {
                    pk[j] = Packet{0ull, 0ull};
                    if (polls && lane + 32 * j < gsize) todo |= 1u << j;
                }
                if (rows)
#pragma unroll
                    for (int u = 0; u < NH; ++u)
                        if (htid + u * T < h) todo |= 256u << u;
                for (unsigned spins = 0; todo; ++spins) {
#pragma unroll
                    for (int j = 0; j < kResSlotPoll; ++j)
                        if ((todo >> j) & 1u) pk[j] = ld_packet(in + (size_t)(lane + 32 * j) * kResSlotBytes);
                    unsigned got = 0;
#pragma unroll
                    for (int u = 0; u < NH; ++u)
                        if (((todo >> u) & 256u) && ld_row(qin + (size_t)(htid + u * T) * RB, tag, hq[u]))
                            got |= 256u << u;
#pragma unroll
                    for (int j = 0; j < kResSlotPoll; ++j)
                        if (((todo >> j) & 1u) && packet_tag(pk[j]) == tag) got |= 1u << j;
                    todo &= ~got;
                    if (spins > P.spin_limit) {
                        atomicOr(P.flags, kFlagBarrierTimeout);
                        s_fail = 1;
                        break;
                    }
                    if ((spins & 1023u) == 1023u && (*(volatile unsigned*)P.flags & kFlagBarrierTimeout)) {
                        s_fail = 1;
                        break;
                    }
                }
                __syncwarp();
                if (polls) {
                    double t = 0.0;
                    unsigned w = 0;
#pragma unroll
                    for (int j = 0; j < kResSlotPoll; ++j)
                        if (lane + 32 * j < gsize) {
                            t += __longlong_as_double((long long)pk[j].lo);
                            w |= (unsigned)pk[j].hi;
                        }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                    if (lane == 0) sh_sum[gen & 1u][sum] = t;
                    if (w) atomicOr(&sh_gbits[gen % 3u], w);
                }
                __syncthreads();
#pragma unroll
                for (int k = 0; k < kResSums; ++k) v[k] = sh_sum[gen & 1u][k];
                bits = sh_gbits[gen % 3u];
                if (tid == 0) sh_gbits[(gen + 2u) % 3u] = 0u;
                timed_out = s_fail != 0;
            }
        }
        if (timed_out) break;
        if constexpr (FS) {
            v[0] = as_float_sum(v[0]);
            v[3] = as_float_sum(v[3]);
        }

        double beta;
        if (turn == kEnd) {
            if (ran) residual = (isfinite(v[0]) && v[0] >= 0.0) ? sqrt(v[0]) : (double)INFINITY;
            const bool solved = have_x && !(bits & 1u);
            if (!have_x && !(fl & kFlagBreakdown)) fl |= kFlagInvalidRhs;
            if (have_x && (bits & 1u)) fl |= kFlagNonFiniteDv;
            if (solved) fl |= kFlagSolved;
            if (solved && P.integrate) {
                if (bits & 2u) {
                    fl |= kFlagIntegrateAbort;
                } else {
#pragma unroll
                    for (int p = 0; p < R; ++p)
                        if (has[p] && cidx[p] >= 0) {
                            st3(P.node_v, node[p], nv[p]);
                            st3(P.node_x, node[p], nx[p]);
                        }
                    fl |= kFlagIntegrated;
                }
            }
            if (converged) fl |= kFlagConverged;
            break;
        } else if (turn == kFirst) {
            delta = v[3];
            turn = kEnd;
            if (bits & 4u) {  // a malformed layout: report, do not solve
                have_x = false;
                fl |= kFlagBreakdown;
            } else if ((bits & 1u) || P.max_iterations <= 0 || !isfinite(P.tolerance) || P.tolerance <= 0.0) {
                // non-finite rhs or invalid settings: the reference clears x (the solve fails)
                have_x = false;
                fl |= kFlagInvalidRhs;
            } else if (!(bits & 2u) && isfinite(delta) && delta >= 0.0) {
                // (else the preconditioner's output is not finite: x stays 0)
                target = P.tolerance * P.tolerance * delta;
                if (isfinite(target)) {
                    ran = true;
                    if (delta <= target)
                        converged = true;
                    else
                        turn = kProducts;
                }
            }
            continue;  // (the exchange's barrier ordered the window's first d)
        } else if (turn == kProducts) {
            turn = kEnd;
            if (pending) {
                if (!close(v[3], bits & 2u, it)) {
                    converged = delta <= target;
                    continue;
                }
                if (delta <= target) {
                    converged = true;
                    continue;
                }
            }
            // One reciprocal for both scalars: alpha = delta / dq (corrected to the quotient),
            // and beta = (r'.s') / delta with r'.s' predicted, which is 1 + (alpha q.z - (q.s
            // + r.z)) / dq.
            const double dq = v[0], inv = 1.0 / dq;
            double alpha = delta * inv;
            alpha = fma(fma(-alpha, dq, delta), inv, alpha);
            if ((bits & 1u) || !isfinite(dq) || dq <= 0.0 || !(FS ? fabs(alpha) <= scalar_max<FS>() : isfinite(alpha))) {
                fl |= kFlagBreakdown;
                converged = delta <= target;
                continue;
            }
            // r'.s' before r' exists; not where it cancels, near the target or at the cap.
            const double slope = fma(alpha, v[2], -v[1]);
            beta = fma(slope, inv, 1.0);
            const double next = fma(alpha, slope, delta);
            pending = next > 0.0625 * delta && next > 1.05 * target && isfinite(next) && isfinite(beta) &&
                      it + 1 < P.max_iterations;
            const Scale<Real> pa(alpha), na = pa.negated();
            sbad = 0;
            rs_next = 0.0;
#pragma unroll
            for (int p = 0; p < R; ++p)
                if (has[p]) {
                    xv[p] = pa.axpy(dv[p], xv[p]);
                    rv[p] = na.axpy(qv[p], rv[p]);
                    sv[p] = apply_minv(mi[p], rv[p]);
                    if (!finite3(sv[p])) sbad = 2u;
                    const double rs = dot_acc<double>(rv[p], sv[p]);
                    rs_next = p == 0 ? rs : rs_next + rs;
                }
#pragma unroll
            for (int u = 0; u < NH; ++u) {
                const int j = htid + u * T;
                if (j < h) {
                    V3<Real> r{hr[j], hr[h + j], hr[2 * h + j]};
                    r = na.axpy(hq[u], r);
                    hr[j] = r.x;
                    hr[h + j] = r.y;
                    hr[2 * h + j] = r.z;
                    Real hmi[9];
#pragma unroll
                    for (int e = 0; e < 9; ++e) hmi[e] = hm[(size_t)e * h + j];
                    hs[u] = apply_minv(hmi, r);
                }
            }
            if (!pending) {
                turn = kConfirm;
                continue;
            }
        } else {
            turn = kEnd;
            const double old = delta;
            if (!close(v[3], bits & 2u, it + 1) || it + 1 >= P.max_iterations || delta <= target) {
                converged = delta <= target;
                continue;
            }
            beta = delta / old;
        }
        // d = s + beta d: the owned row, then the halo copies.
        const Real bt = Real(beta);
#pragma unroll
        for (int p = 0; p < R; ++p)
            if (has[p]) {
                dv[p] = fma3(bt, dv[p], sv[p]);
                Real* d = win + 3 * (tid + p * T);
                d[0] = dv[p].x;
                d[1] = dv[p].y;
                d[2] = dv[p].z;
            }
#pragma unroll
        for (int u = 0; u < NH; ++u) {
            const int j = htid + u * T;
            if (j < h) {
                Real* d = win + 3 * (m + j);
                const V3<Real> nd = fma3(bt, V3<Real>{d[0], d[1], d[2]}, hs[u]);
                d[0] = nd.x;
                d[1] = nd.y;
                d[2] = nd.z;
            }
        }
        ++it;
        turn = kProducts;
        __syncthreads();
    }

    if (timed_out) fl |= kFlagBarrierTimeout;
    if (leader && tid == 0) {
        // The next solve's tags start after every tag a block of this group may have used
        // (after a timeout a block may be an exchange ahead).
        if (!CL && gsize > 1) P.epoch[gfirst] = epoch + gen + 16u;
        if (P.grouped) {
            // Per body; world-wide: the largest iteration count and residual, the OR of the
            // failure flags and the AND of the success flags (missing: what some body lacks).
            bs->iterations = iterations;
            bs->converged = converged ? 1 : 0;
            bs->residual_norm = residual;
            bs->flags = fl;
            atomicMax(&P.stats->iterations, iterations);
            if (residual >= 0.0)  // non-negative doubles order like their bit patterns
                atomicMax(reinterpret_cast<unsigned long long*>(&P.stats->residual_norm),
                          (unsigned long long)__double_as_longlong(residual));
            atomicOr(P.flags, fl & ~(kFlagSolved | kFlagIntegrated | kFlagConverged));
            if (!(fl & kFlagSolved)) atomicOr(P.missing, kFlagSolved);
            if (!(fl & kFlagIntegrated)) atomicOr(P.missing, kFlagIntegrated);
            if (!(fl & kFlagConverged)) atomicOr(P.missing, kFlagConverged);
        } else {
            P.stats->iterations = iterations;
            P.stats->converged = converged ? 1 : 0;
            P.stats->residual_norm = residual;
            atomicOr(P.flags, fl);
        }
    } else if (timed_out && tid == 0) {
        atomicOr(P.flags, kFlagBarrierTimeout);
    }
    if (TM && tslots > 0) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512u) : "memory");
        }
    }
    if (CL) cluster_barrier();  // nobody's shared memory goes while a peer may still write to it
}

template <class Real, bool FS>
const void* res_kernel(int threads, bool cluster, int rpt, bool tmem)
{
    if (cluster)
        return threads <= 256 ? (const void*)pcg_res_kernel<Real, 256, true, 1, false, FS>
                              : (const void*)pcg_res_kernel<Real, 512, true, 1, false, FS>;
    if (rpt == 1 && threads <= 256) {
        if constexpr (sizeof(Real) == 8)
            if (tmem) return (const void*)pcg_res_kernel<Real, 256, false, 1, true, FS>;
        return (const void*)pcg_res_kernel<Real, 256, false, 1, false, FS>;
    }
    if constexpr (sizeof(Real) == 4)
        return (const void*)pcg_res_kernel<Real, kResPairThreads, false, 2, true, FS>;  // (never asked for 512 threads)
    else
        return (const void*)pcg_res_kernel<Real, 512, false, 1, false, FS>;
}
template <class Real>
const void* res_kernel(int threads, bool cluster, int rpt, bool tmem, bool float_sums)
{
    if constexpr (sizeof(Real) == 4)
        if (float_sums) return res_kernel<Real, true>(threads, cluster, rpt, tmem);
    return res_kernel<Real, false>(threads, cluster, rpt, tmem);
}

template <class Real>
ResLimits query_limits(int dev)
{
    ResLimits lim;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return lim;
    int per_sm = 1 << 20;
    struct {
        int threads, rpt;
        bool cluster, tmem;
    } const kinds[] = {{256, 1, false, false}, {256, 1, false, true}, {256, 1, true, false}, {512, 1, true, false},
                       {sizeof(Real) == 4 ? kResPairThreads : 512, sizeof(Real) == 4 ? 2 : 1, false, false}};
    for (int i = 0; i < 2 * int(sizeof(kinds) / sizeof(kinds[0])); ++i) {
        const auto& kind = kinds[i / 2];
        const void* k = res_kernel<Real>(kind.threads, kind.cluster, kind.rpt, kind.tmem, i % 2 != 0);
        int b = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmemLimit) != cudaSuccess ||
            (kind.cluster && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, kind.threads, kResSmemLimit) != cudaSuccess)
            return lim;
        per_sm = b < per_sm ? b : per_sm;
    }
    lim.blocks = sms * per_sm;
    for (int q = 0; q < 5; ++q) {
        lim.clusters[q] = 1 << 20;
        for (const int threads : {256, 512}) {
            cudaLaunchConfig_t c{};
            c.gridDim = dim3(1u << q);
            c.blockDim = dim3((unsigned)threads);
            c.dynamicSmemBytes = kResSmemLimit;
            cudaLaunchAttribute a;
            a.id = cudaLaunchAttributeClusterDimension;
            a.val.clusterDim.x = 1u << q;
            a.val.clusterDim.y = a.val.clusterDim.z = 1;
            c.attrs = &a;
            c.numAttrs = 1;
            int k = 0;
            if (cudaOccupancyMaxActiveClusters(&k, res_kernel<Real>(threads, true, 1, false, false), &c) != cudaSuccess) {
                cudaGetLastError();
                k = 0;
            }
            lim.clusters[q] = k < lim.clusters[q] ? k : lim.clusters[q];
        }
    }
    return lim;
}

}  // namespace

// A device's limits do not change: asked once per device (the queries take milliseconds),
// which also raises the kernels' shared-memory limits on it.
template <class Real>
ResLimits pcg_res_limits()
{
    constexpr int kDevices = 64;
    static std::once_flag asked[kDevices];
    static ResLimits limits[kDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return ResLimits{};
    std::call_once(asked[dev], [dev] { limits[dev] = query_limits<Real>(dev); });
    return limits[dev];
}

template <class Real>
cudaError_t launch_pcg_res_kernel(const ResPcgArgs<Real>& args, int threads, int rpt, int cluster, int grid,
                                  cudaStream_t stream)
{
    ResPcgArgs<Real> a = args;
    void* kargs[] = {&a};
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = args.smem_bytes;
    c.stream = stream;
    cudaLaunchAttribute at;
    if (cluster > 0) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)cluster;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelExC(&c, res_kernel<Real>(threads, cluster > 0, rpt, args.tmem_slots > 0, args.float_sums != 0),
                                kargs);
}

template cudaError_t launch_pcg_res_kernel<float>(const ResPcgArgs<float>&, int, int, int, int, cudaStream_t);
template cudaError_t launch_pcg_res_kernel<double>(const ResPcgArgs<double>&, int, int, int, int, cudaStream_t);
template ResLimits pcg_res_limits<float>();
template ResLimits pcg_res_limits<double>();

}  // namespace pk
