// pk_pcg_part.cu -- the part-resident cooperative block-Jacobi PCG kernel for coupled solves
// of systems whose matrix exceeds the chip (pk_pcg_res.cu) and whose parts fit its windows.
//
// The solve of the other PCG kernels (SolvePreconditionedConjugateGradient,
// src/Core/Solvers/Linear/ConjugateGradientSolver.cpp:114-241, with the SpMV of
// SparseBlockMatrix::Multiply, src/Math/SparseBlockMatrix.cpp:209-268, and
// World::IntegrateImplicitEuler, src/Core/World/World.cpp:644-695, fused at the end), laid
// out as pk_pcg_slab.cu (which keeps the per-body solves and the symmetric stream): one block
// per part, the search directions of its window (rows, then halo) in shared memory, full
// symmetric rows streamed by TMA bulk copies into a ring, x and r (in FP32 M^-1 too) of a row
// in tensor memory.  What differs:
//
// * one exchange per iteration with the predicted beta of pk_pcg_res.cu; the rows of d that
//   other windows hold are pushed as tagged packets and collected by the halo warp while the
//   consumers stream the interior tiles.
// * a tile's values go to registers first (a row of up to 16 blocks is one pass of its lanes)
//   and the stage is free again before they are multiplied: the three consumer groups would
//   otherwise hold three of the five FP64 stages that fit beside a window of 5,300 rows (138
//   against 117 us an iteration).
// * the producer warp runs on its own, outside the block's barriers.
// * FP64: M^-1 is read from global memory (part order, nine arrays), two rows at a time.
//
// Per iteration, FP64 against the ring kernel: 51,450 rows 27.9 -> 15.8 us, 126 k rows 51.6 ->
// 29.7, 537 k rows 177.5 -> 117.  FP32 against pcg_slab_kernel: 122,400 rows 22.4 -> 17.6,
// 199,836 rows 29.3 -> 23.7, 537 k rows 55.6 -> 55.1.  Large FP32 systems are bound by the
// stream (DRAM), the others by a tile's latency in its consumer warps and by the exchange,
// whose packets queue behind the ring's refill; holding the refill back until the update is
// done was slower (57.4 us at 537 k rows), a ring of nine stages too (17.9 at 122,400).
//
// All sums keep one fixed order; every wait is bounded and the kernel leaves through its
// normal exit, after waiting for its own bulk copies.  No TMA multicast is used.
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "pk_device.cuh"
#include "pk_exchange.cuh"

namespace pk {
namespace {

constexpr int kConsumerWarps = 12, kGroups = 3, kGroupWarps = 4;
constexpr int kTeamWarps = kConsumerWarps + 1;     // and the halo warp; the producer runs alone
constexpr int kPartThreads = 32 * (kConsumerWarps + 2);
constexpr int kOwners = 32 * kConsumerWarps;       // record k of thread t: row t + 384 k
constexpr unsigned kOwnBar = 1, kTeamBar = 2;      // named barriers

__device__ __forceinline__ void mbar_arrive_one(unsigned long long* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Bulk copy global -> shared, evicted first from L2 (the stream must not push the vectors out).
__device__ __forceinline__ void bulk_g2s_first(void* dst, const void* src, unsigned bytes, unsigned long long* bar,
                                               unsigned long long pol)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
            "r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(pol)
        : "memory");
}

static_assert(kTagSlotBytes == kResSlotBytes, "the host sizes the inboxes");

// A row record of sixteen 32-bit columns: x and r, in FP32 then M^-1 (column-major).
struct Rec {
    unsigned w[16];
};
#define PK_IO(c) c(t.w[0]), c(t.w[1]), c(t.w[2]), c(t.w[3]), c(t.w[4]), c(t.w[5]), c(t.w[6]), c(t.w[7]), c(t.w[8]), \
                 c(t.w[9]), c(t.w[10]), c(t.w[11]), c(t.w[12]), c(t.w[13]), c(t.w[14]), c(t.w[15])
__device__ __forceinline__ void rec_ld(unsigned addr, Rec& t)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : PK_IO("=r")
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void rec_st(unsigned addr, const Rec& t)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::PK_IO("r"),
        "r"(addr)
        : "memory");
}
#undef PK_IO
__device__ __forceinline__ float rec_at(const Rec& t, int i, float) { return __uint_as_float(t.w[i]); }
__device__ __forceinline__ double rec_at(const Rec& t, int i, double)
{
    return __hiloint2double((int)t.w[2 * i + 1], (int)t.w[2 * i]);
}
__device__ __forceinline__ void rec_set(Rec& t, int i, float v) { t.w[i] = __float_as_uint(v); }
__device__ __forceinline__ void rec_set(Rec& t, int i, double v)
{
    t.w[2 * i] = (unsigned)__double2loint(v);
    t.w[2 * i + 1] = (unsigned)__double2hiint(v);
}
template <class Real>
__device__ __forceinline__ V3<Real> rec_get(const Rec& t, int o)  // 0: x, 3: r
{
    return V3<Real>{rec_at(t, o, Real()), rec_at(t, o + 1, Real()), rec_at(t, o + 2, Real())};
}
template <class Real>
__device__ __forceinline__ void rec_put(Rec& t, int o, V3<Real> v)
{
    rec_set(t, o, v.x);
    rec_set(t, o + 1, v.y);
    rec_set(t, o + 2, v.z);
}
__device__ __forceinline__ V3<float> ld_q(const float* p)
{
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p));
    return V3<float>{a.x, a.y, a.z};
}
__device__ __forceinline__ void st_q(float* p, V3<float> v)
{
    __stcg(reinterpret_cast<float4*>(p), make_float4(v.x, v.y, v.z, 0.f));
}
__device__ __forceinline__ V3<double> ld_q(const double* p)
{
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    return V3<double>{a.x, a.y, __ldcg(p + 2)};
}
__device__ __forceinline__ void st_q(double* p, V3<double> v)
{
    __stcg(reinterpret_cast<double2*>(p), make_double2(v.x, v.y));
    __stcg(p + 2, v.z);
}

// FS: the sums judged as floats (as_float_sum).
template <class Real, bool FS>
__global__ void __launch_bounds__(kPartThreads, 1) pcg_part_kernel(const __grid_constant__ PartPcgArgs<Real> P)
{
    constexpr bool kWide = sizeof(Real) == 8;
    constexpr int LPR = kWide ? kWideLanes : kSlabLanesPerRow, NE = 16 / LPR;  // entries of a lane and pass
    constexpr int kEntryBytes = kWide ? kWideEntryBytes : kSlabEntryBytes, kValueBytes = 9 * (int)sizeof(Real);
    constexpr int kCapE = kWide ? kWideCapE : kSlabCapE, kRows = kWide ? kWideRows : kSlabRows;
    constexpr int kStageBytes = kWide ? kWideStageBytes : kSlabStageBytes;
    constexpr int kMaxTiles = kWide ? kWideMaxTiles : kSlabMaxTiles;
    constexpr int kRowBytes = kWide ? 32 : 16;  // packets of a pushed row
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) unsigned long long full_bar[kPartMaxStages];
    __shared__ __align__(8) unsigned long long empty_bar[kPartMaxStages];
    __shared__ TagShared sh;
    __shared__ int s_fail, s_bad, s_done, s_halo_gen;
    __shared__ unsigned s_tmem;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x;
    const bool consumer = warp < kConsumerWarps, halo_warp = warp == kConsumerWarps;
    const bool producer = warp == kConsumerWarps + 1;
    const TagTeam team{kTeamWarps, kTeamBar};
    const int group = warp / kGroupWarps;
    const int slot_row = ((warp % kGroupWarps) * 32 + lane) / LPR, sub = lane % LPR;
    const int S = min(P.stages, kPartMaxStages);
    Real* const win = reinterpret_cast<Real*>(dyn);  // 3 values per window row
    unsigned char* const ring = dyn + P.ring_offset;
    int4* const table = reinterpret_cast<int4*>(ring + (size_t)S * kStageBytes);

    const unsigned in_flags = *(volatile unsigned*)P.flags;
    const bool skip = P.skip_on_flags && (in_flags & (kFlagPrecomputeFailed | kFlagSingularDiag));
    if (skip) {
        if (blk == 0 && tid == 0) {
            P.stats->iterations = 0;
            P.stats->converged = 0;
            P.stats->residual_norm = 0.0;
        }
        return;
    }
    // The part: rows [row0, row0 + m) of the slab order, halo rows from halo0, tiles from tile0,
    // sends from send0.  A part that does not fit (the host never builds one) is emptied and
    // reports a breakdown.
    const int* pi = P.part_info + (size_t)kSlabPartInts * blk;
    int row0 = __ldg(pi), m = __ldg(pi + 1), halo0 = __ldg(pi + 2), h = __ldg(pi + 3), tile0 = __ldg(pi + 4),
        ntiles = __ldg(pi + 5), send0 = __ldg(P.send_start + blk), sends_n = __ldg(P.send_start + blk + 1) - send0;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], kGroupWarps);
        }
        mbar_fence_init();
        tag_init(sh);
        s_fail = s_bad = s_done = s_halo_gen = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (m < 0 || m > kSlabMaxRows || h < 0 || m + h > P.win_cap || row0 < 0 || row0 + m > P.n || ntiles < 0 ||
        ntiles > kMaxTiles || halo0 < 0 || halo0 + h > P.halo_count || tile0 < 0 ||
        tile0 + ntiles > P.tile_count || sends_n < 0 || send0 < 0 || send0 + sends_n > P.halo_count) {
        m = h = ntiles = sends_n = row0 = halo0 = 0;
        if (tid == 0) s_bad = 1;
    }
    const int wn = m + h;
    // Tile descriptors, checked once: a bad one becomes an empty tile and reports a breakdown.
    for (int i = tid; i < ntiles; i += blockDim.x) {
        int4 d = __ldg(P.tile_desc + tile0 + i);
        const int ne = (d.y - kSlabHeaderBytes) / kEntryBytes;
        if (!(d.x >= 0 && d.y >= kSlabHeaderBytes && d.y <= kStageBytes && (d.y & 15) == 0 &&
              d.y == kSlabHeaderBytes + kEntryBytes * ne && ne <= kCapE && d.w >= 1 &&
              d.w <= kRows && d.z >= 0 && d.z + d.w <= m &&
              16ull * (unsigned long long)d.x + (unsigned long long)d.y <= P.stream_bytes)) {
            d = make_int4(0, 0, 0, 0);
            s_bad = 1;
        }
        table[i] = d;
    }
    __syncthreads();

    const int rt = tid;
    const int krows = consumer ? (m + kOwners - 1) / kOwners : 0;
    const unsigned tmem0 =
        s_tmem + ((32u * (unsigned)(warp % 4)) << 16) + (unsigned)((warp / 4) * kSlabRowsPerThread * 16);
    unsigned issued = 0;  // tiles issued so far (producer lane 0)
    unsigned xgen = 0;
    const V3<Real> zero{Real(0), Real(0), Real(0)};
    // Ring position p is stage p % S in its use p / S, counted along; the iteration's first:
    int bstage = 0;
    unsigned buse = 0;
    const int dstage = ntiles % S;
    const unsigned duse = (unsigned)(ntiles / S);

    auto produce = [&]() {
        unsigned long long pol;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
        int stage = 0, tile = 0;
        unsigned use = 0;
        for (;;) {
            const int4 d = table[tile];
            for (unsigned long long spins = 0; use > 0 && !mbar_try_wait(&empty_bar[stage], (use - 1) & 1u); ++spins) {
                if (*(volatile int*)&s_done) return;
                if (spins > kBarrierSpinLimit) {
                    s_fail = 1;
                    return;
                }
            }
            if (*(volatile int*)&s_done) return;
            mbar_arrive_expect_tx(&full_bar[stage], (unsigned)d.y);
            if (d.y > 0)
                bulk_g2s_first(ring + (size_t)stage * kStageBytes, P.stream + 16 * (size_t)d.x, (unsigned)d.y,
                               &full_bar[stage], pol);
            ++issued;
            if (++tile == ntiles) tile = 0;
            if (++stage == S) {
                stage = 0;
                ++use;
            }
        }
    };

    // The window's halo rows pushed with `tag` (halo warp).
    auto collect_halo = [&](unsigned tag) {
        constexpr int B = 4;  // rows of a poll, all loads in flight
        const unsigned char* in = P.rows_in + (size_t)halo0 * kRowBytes;
        for (int w0 = lane; w0 < h; w0 += B * 32) {
            unsigned todo = 0;
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (w0 + u * 32 < h) todo |= 1u << u;
            for (unsigned spins = 0; todo; ++spins) {
                V3<Real> v[B];
                unsigned got = 0;
#pragma unroll
                for (int u = 0; u < B; ++u)
                    if (((todo >> u) & 1u) && ld_row(in + (size_t)(w0 + u * 32) * kRowBytes, tag, v[u])) got |= 1u << u;
#pragma unroll
                for (int u = 0; u < B; ++u)
                    if ((got >> u) & 1u) {
                        Real* d = win + 3 * (m + w0 + u * 32);
                        d[0] = v[u].x;
                        d[1] = v[u].y;
                        d[2] = v[u].z;
                    }
                todo &= ~got;
                if (spins > P.spin_limit) {
                    atomicOr(P.flags, kFlagBarrierTimeout);
                    s_fail = 1;
                    return;
                }
                if ((spins & 1023u) == 1023u && (*(volatile unsigned*)P.flags & kFlagBarrierTimeout)) {
                    s_fail = 1;
                    return;
                }
            }
        }
    };

    // Phase A: q = A d for the part's rows, to global memory.
    auto phase_a = [&](int it, double& dq, unsigned& bits) {
        if (halo_warp) {
            collect_halo((unsigned)it + 1u);
            __syncwarp();
            if (lane == 0) {
                __threadfence_block();
                *(volatile int*)&s_halo_gen = it + 1;
            }
        } else {
            const int wmax = max(wn - 1, 0);
            bool halo_in = false;
            int s = bstage + group;
            unsigned u = buse;
            if (s >= S) {
                s -= S;
                ++u;
            }
            for (int t = group; t < ntiles; t += kGroups) {
                // The stage's earlier tile may be another group's, not even landed: its phase
                // must be over before this one's parity says anything.
                if ((u > 0 && !mbar_wait(&empty_bar[s], (u - 1) & 1u)) || !mbar_wait(&full_bar[s], u & 1u)) {
                    s_fail = 1;
                    break;
                }
                const int4 d = table[t];
                const unsigned char* st = ring + (size_t)s * kStageBytes;
                const int ne = d.y > 0 ? (d.y - kSlabHeaderBytes) / kEntryBytes : 0;
                const unsigned short* roff = reinterpret_cast<const unsigned short*>(st);
                const Real* vals = reinterpret_cast<const Real*>(st + kSlabHeaderBytes);
                const unsigned short* lcol = reinterpret_cast<const unsigned short*>(st + kSlabHeaderBytes + kValueBytes * ne);
                const bool valid = slot_row < d.w, flagged = d.y > 0 && roff[kSlabHaloWord] != 0;
                int e0 = 0, e1 = 0;
                if (valid) {
                    e0 = min((int)roff[slot_row], ne);
                    e1 = min((int)roff[slot_row + 1], ne);
                }
                V3<Real> acc = zero;
                // sixteen entries of a row a pass, the stage released after the last pass's loads
                const int passes = __reduce_max_sync(0xffffffffu, (e1 - e0 + 15) / 16);
                for (int p = 0; p < passes || p == 0; ++p) {
                    int c[NE];
                    Real b[NE][9];
                    bool live[NE];
#pragma unroll
                    for (int q = 0; q < NE; ++q) {
                        const int j = e0 + sub + (NE * p + q) * LPR;
                        live[q] = j < e1;
                        c[q] = live[q] ? 3 * min((int)lcol[j], wmax) : 0;
#pragma unroll
                        for (int e = 0; e < 9; ++e) b[q][e] = live[q] ? vals[9 * j + e] : Real(0);
                    }
                    if (p + 1 >= passes) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive_one(&empty_bar[s]);
                    }
                    // the first tile with a halo column waits until the halo warp has filled it
                    if (flagged && !halo_in) {
                        if (!wait_shared(&s_halo_gen, it + 1)) s_fail = 1;
                        halo_in = true;
                    }
#pragma unroll
                    for (int q = 0; q < NE; ++q)
                        if (live[q]) {
                            const Real x = win[c[q]], y = win[c[q] + 1], z = win[c[q] + 2];
                            acc.x += b[q][0] * x + b[q][3] * y + b[q][6] * z;
                            acc.y += b[q][1] * x + b[q][4] * y + b[q][7] * z;
                            acc.z += b[q][2] * x + b[q][5] * y + b[q][8] * z;
                        }
                }
                s += kGroups;
                if (s >= S) {
                    s -= S;
                    ++u;
                }
#pragma unroll
                for (int off = LPR / 2; off > 0; off >>= 1) {
                    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
                    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
                    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, off);
                }
                if (valid && sub == 0) {
                    const int li = d.z + slot_row;
                    st_q(P.qs + 4 * (size_t)(row0 + li), acc);
                    dq += dot_acc<double>(V3<Real>{win[3 * li], win[3 * li + 1], win[3 * li + 2]}, acc);
                    if (!finite3(acc)) bits |= 1u;
                }
            }
        }
        bstage += dstage;
        buse += duse;
        if (bstage >= S) {
            bstage -= S;
            ++buse;
        }
    };

    // f(k, local row or -1, its q, its M^-1, its record) for the thread's rows, the loads of two in flight.
    auto each_row = [&](bool want_q, auto&& f) {
        for (int k0 = 0; k0 < krows; k0 += 2) {
            V3<Real> q[2] = {zero, zero};
            Real mi[2][9];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = rt + kOwners * (k0 + u);
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    mi[u][e] = kWide && i < m ? __ldcg(P.mrow + (size_t)e * P.n + row0 + i) : Real(0);
                if (want_q && i < m) q[u] = ld_q(P.qs + 4 * (size_t)(row0 + i));
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (k0 + u >= krows) break;
                const int i = rt + kOwners * (k0 + u);
                __syncwarp();
                Rec rec;
                rec_ld(tmem0 + 16u * (unsigned)(k0 + u), rec);
                if (!kWide) {
#pragma unroll
                    for (int e = 0; e < 9; ++e) mi[u][e] = rec_at(rec, 6 + e, Real());
                }
                f(k0 + u, i < m ? i : -1, q[u], mi[u], rec);
            }
        }
    };
    auto put_d = [&](int i, V3<Real> v) {
        win[3 * i] = v.x;
        win[3 * i + 1] = v.y;
        win[3 * i + 2] = v.z;
    };
    auto get_d = [&](int i) { return V3<Real>{win[3 * i], win[3 * i + 1], win[3 * i + 2]}; };
    // The rows of d that other parts' windows hold, once all own rows are written (which the
    // consumers' reads wait for too).
    auto push_rows = [&](unsigned tag) {
        if (!consumer) return;
        int2 next[2];  // loaded while the barrier completes
#pragma unroll
        for (int u = 0; u < 2; ++u)
            next[u] = rt + u * kOwners < sends_n ? __ldg(P.send + send0 + rt + u * kOwners) : make_int2(-1, -1);
        asm volatile("bar.sync %0, %1;" ::"r"(kOwnBar), "r"(kOwners) : "memory");
        auto push = [&](int2 e) {
            if ((unsigned)e.x < (unsigned)m && (unsigned)e.y < (unsigned)P.halo_count)
                st_row(P.rows_in + (size_t)e.y * kRowBytes, get_d(e.x), tag);
        };
        push(next[0]);
        push(next[1]);
        for (int e = rt + 2 * kOwners; e < sends_n; e += kOwners) push(__ldg(P.send + send0 + e));
    };
    auto exchange = [&](double (&v)[kTagSums], unsigned& bits) {
        const bool ok = tag_exchange(P.sums_in, (int)gridDim.x, blk, ++xgen, v, bits, kConsumerWarps, P.flags, team, sh);
        if constexpr (FS) {
            v[0] = as_float_sum(v[0]);
            v[3] = as_float_sum(v[3]);
        }
        return ok;
    };

    unsigned fl = 0, sbad = 0;
    int iterations = 0;
    bool converged = false, have_x = true, ran = false, timed_out = false;
    double residual = 0.0, delta = 0.0, target = 0.0, rs_next = 0.0;
    if (producer) {
        if (lane == 0 && ntiles > 0) produce();
        __syncwarp();
        goto finish;
    }
    {
        // x = 0, r = b, M^-1 in part order; d = s = M^-1 r in the window; r.s, finiteness.
        double v[kTagSums] = {0.0, 0.0, 0.0, 0.0};
        unsigned bad = s_bad ? 4u : 0u;
        for (int k = 0; k < krows; ++k) {
            const int i = rt + kOwners * k;
            Rec rec{};
            if (i < m) {
                int c = __ldg(P.perm + row0 + i);
                if ((unsigned)c >= (unsigned)P.n) {
                    c = 0;
                    bad |= 4u;
                }
                const V3<Real> b = ld3(P.b, c);
                Real mi[9];
                bool fin = true;
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    mi[e] = __ldg(P.minv + 9 * (size_t)c + e);
                    fin = fin && isfinite(mi[e]);
                    if constexpr (kWide)
                        __stcg(P.mrow + (size_t)e * P.n + row0 + i, mi[e]);
                    else
                        rec_set(rec, 6 + e, mi[e]);
                }
                const V3<Real> s = apply_minv(mi, b);
                if (!finite3(b)) bad |= 1u;
                if (!fin || !finite3(s)) bad |= 2u;
                rec_put(rec, 3, b);
                put_d(i, s);
                rs_next += dot_acc<double>(b, s);
            }
            __syncwarp();
            rec_st(tmem0 + 16u * (unsigned)k, rec);
        }
        push_rows(1u);
        v[3] = rs_next;
        if (!exchange(v, bad)) {
            timed_out = true;
            goto finish;
        }
        delta = v[3];
        if (bad & 4u) {  // a malformed layout: report, do not solve
            have_x = false;
            fl |= kFlagBreakdown;
            goto final_check;
        }
        // non-finite rhs or invalid settings: the reference clears x (the solve fails)
        if ((bad & 1u) || P.max_iterations <= 0 || !isfinite(P.tolerance) || P.tolerance <= 0.0) {
            have_x = false;
            fl |= kFlagInvalidRhs;
            goto final_check;
        }
        if (bad & 2u) goto final_check;  // preconditioner output not finite: x stays 0
        if (!isfinite(delta) || delta < 0.0) goto final_check;
        target = P.tolerance * P.tolerance * delta;
        if (!isfinite(target)) goto final_check;
    }
    ran = true;
    if (delta <= target) {
        converged = true;
        goto final_check;
    }
    {
        // The end of an iteration whose r.s is known: false ends the solve.
        auto close = [&](double new_delta, unsigned broken, int done) -> bool {
            if (broken) {
                fl |= kFlagBreakdown;
                return false;
            }
            const double old = delta;
            delta = new_delta;
            // (the last test: delta / old overflows)
            if (!isfinite(delta) || !isfinite(old) || old <= 0.0 ||
                (old < 1.0 && fabs(delta) > scalar_max<FS>() * old)) {
                fl |= kFlagBreakdown;
                return false;
            }
            iterations = done;
            return true;
        };
        bool pending = false;  // the last iteration's r.s comes with the next exchange
        for (int it = 0;; ++it) {
            double v[kTagSums] = {0.0, 0.0, 0.0, 0.0};
            unsigned bits = sbad;
            phase_a(it, v[0], bits);
            if (s_fail) bits |= 8u;
            team.sync();  // q of all rows is written
            each_row(true, [&](int, int i, V3<Real> q, const Real(&mi)[9], Rec& rec) {
                if (i < 0) return;
                const V3<Real> r = rec_get<Real>(rec, 3), s = apply_minv(mi, r), z = apply_minv(mi, q);
                v[1] += dot_acc<double>(q, s) + dot_acc<double>(r, z);
                v[2] += dot_acc<double>(q, z);
            });
            v[3] = rs_next;
            if (!exchange(v, bits) || (bits & 8u)) {
                timed_out = true;
                goto finish;
            }
            if (pending) {
                if (!close(v[3], bits & 2u, it)) break;
                if (delta <= target) break;
            }
            // alpha, and beta with r'.s' predicted (pk_pcg_res.cu)
            const double dq = v[0], inv = 1.0 / dq;
            double alpha = delta * inv;
            alpha = fma(fma(-alpha, dq, delta), inv, alpha);
            if ((bits & 1u) || !isfinite(dq) || dq <= 0.0 || !(FS ? fabs(alpha) <= scalar_max<FS>() : isfinite(alpha))) {
                fl |= kFlagBreakdown;
                break;
            }
            const double slope = fma(alpha, v[2], -v[1]);
            double beta = fma(slope, inv, 1.0);
            const double next = fma(alpha, slope, delta);
            pending = next > 0.0625 * delta && next > 1.05 * target && isfinite(next) && isfinite(beta) &&
                      it + 1 < P.max_iterations;
            sbad = 0;
            rs_next = 0.0;
            // x += alpha d, r -= alpha q, s = M^-1 r; with the prediction also d = s + beta d.
            const Scale<Real> pa(alpha), na = pa.negated();
            const Real bt = Real(beta);
            each_row(true, [&](int k, int i, V3<Real> q, const Real(&mi)[9], Rec& rec) {
                if (i >= 0) {
                    const V3<Real> d = get_d(i), r = na.axpy(q, rec_get<Real>(rec, 3)), s = apply_minv(mi, r);
                    rec_put(rec, 0, pa.axpy(d, rec_get<Real>(rec, 0)));
                    rec_put(rec, 3, r);
                    if (!finite3(s)) sbad = 2u;
                    rs_next += dot_acc<double>(r, s);
                    if (pending) put_d(i, fma3(bt, d, s));
                }
                __syncwarp();
                rec_st(tmem0 + 16u * (unsigned)k, rec);
            });
            if (!pending) {
                double w[kTagSums] = {0.0, 0.0, 0.0, rs_next};
                unsigned wb = sbad;
                if (!exchange(w, wb)) {
                    timed_out = true;
                    goto finish;
                }
                const double old = delta;
                if (!close(w[3], wb & 2u, it + 1) || it + 1 >= P.max_iterations || delta <= target) break;
                beta = delta / old;
                sbad = 0;
                const Real bc = Real(beta);
                each_row(false, [&](int, int i, V3<Real>, const Real(&mi)[9], Rec& rec) {
                    if (i >= 0) put_d(i, fma3(bc, get_d(i), apply_minv(mi, rec_get<Real>(rec, 3))));
                });
            }
            push_rows((unsigned)it + 2u);
        }
        converged = delta <= target;
    }

final_check:
    if (tid == 0) *(volatile int*)&s_done = 1;
    // delta-v back in dynamic-row order; the solve succeeds when it is present and finite;
    // integration is all-or-nothing.
    {
        unsigned bad = 0;
        double v[kTagSums] = {0.0, 0.0, 0.0, 0.0};  // v[0]: r.r
        // Two rows at a time: f(record, dynamic row, node, its x, its v).
        auto each_node = [&](auto&& f) {
            for (int k0 = 0; k0 < krows; k0 += 2) {
                int c[2], node[2];
                V3<Real> xo[2] = {zero, zero}, vo[2] = {zero, zero};
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = rt + kOwners * (k0 + u);
                    c[u] = -1;
                    node[u] = 0;
                    if (i >= m) continue;
                    c[u] = __ldg(P.perm + row0 + i);
                    if ((unsigned)c[u] >= (unsigned)P.n) {
                        c[u] = -1;
                        bad |= 1u;
                    } else if (P.integrate) {
                        node[u] = __ldg(P.dyn_to_node + c[u]);
                        xo[u] = ldplain3(P.node_x, node[u]);
                        vo[u] = ldplain3(P.node_v, node[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (k0 + u >= krows) break;
                    Rec rec;
                    __syncwarp();
                    rec_ld(tmem0 + 16u * (unsigned)(k0 + u), rec);
                    if (c[u] >= 0) f(rec, c[u], node[u], xo[u], vo[u]);
                }
            }
        };
        each_node([&](const Rec& rec, int c, int, V3<Real> xo, V3<Real> vo) {
            const V3<Real> dv = have_x ? rec_get<Real>(rec, 0) : zero, r = rec_get<Real>(rec, 3);
            v[0] += dot_acc<double>(r, r);
            st3(P.x, c, dv);
            if (!finite3(dv)) bad |= 1u;
            if (P.integrate) {
                const V3<Real> nv = vo + dv;
                const V3<Real> nx = xo + nv * P.dt;
                if (!finite3(xo) || !finite3(vo) || !finite3(nv) || !finite3(nx)) bad |= 2u;
            }
        });
        if (!exchange(v, bad)) {
            timed_out = true;
            goto finish;
        }
        if (ran) residual = (isfinite(v[0]) && v[0] >= 0.0) ? sqrt(v[0]) : (double)INFINITY;
        const bool solved = have_x && !(bad & 1u);
        if (!have_x && !(fl & kFlagBreakdown)) fl |= kFlagInvalidRhs;
        if (have_x && (bad & 1u)) fl |= kFlagNonFiniteDv;
        if (solved) fl |= kFlagSolved;
        if (solved && P.integrate) {
            if (bad & 2u) {
                fl |= kFlagIntegrateAbort;
            } else {
                each_node([&](const Rec& rec, int, int node, V3<Real> xo, V3<Real> vo) {
                    const V3<Real> nv = vo + rec_get<Real>(rec, 0);
                    const V3<Real> nx = xo + nv * P.dt;
                    st3(P.node_v, node, nv);
                    st3(P.node_x, node, nx);
                });
                fl |= kFlagIntegrated;
            }
        }
        if (converged) fl |= kFlagConverged;
    }

finish:
    if (tid == 0) *(volatile int*)&s_done = 1;
    if (timed_out) fl |= kFlagBarrierTimeout;
    // Bulk copies issued ahead must land before the block exits.
    if (producer && lane == 0) {
        for (unsigned k = 0; k < (unsigned)S && k < issued; ++k) {
            const unsigned p = issued - 1 - k;
            mbar_wait(&full_bar[p % (unsigned)S], (p / (unsigned)S) & 1u);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (blk == 0 && tid == 0) {
        P.stats->iterations = iterations;
        P.stats->converged = converged ? 1 : 0;
        P.stats->residual_norm = residual;
        atomicOr(P.flags, fl);
    } else if (timed_out && tid == 0) {
        atomicOr(P.flags, kFlagBarrierTimeout);
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512u) : "memory");
    }
}

// One block per tile: its header and columns (once, `layout`), or its values: nine doubles an
// entry in stream order, gathered from the entry's upper block (element j = 3 c + i of a
// transposed entry is element 3 i + c of the block; padding entries are zero).  A tile that
// does not match its entry list (the host never builds one) is left alone.
constexpr int kWideFillThreads = 128;
__global__ void __launch_bounds__(kWideFillThreads) wide_fill_kernel(WideFillArgs A)
{
    const int t = blockIdx.x;
    if (t >= A.tile_count) return;
    const int4 d = __ldg(A.tile_desc + t);
    const int e0 = __ldg(A.tile_entry0 + t), ne = __ldg(A.tile_entry0 + t + 1) - e0;
    const unsigned long long at = 16ull * (unsigned long long)d.x;
    if (e0 < 0 || ne <= 0 || e0 + ne > A.entries || d.x < 0 || (ne & 7) != 0 || (e0 & 7) != 0 ||
        d.y != kSlabHeaderBytes + kWideEntryBytes * ne || at + (unsigned long long)d.y > A.stream_bytes)
        return;
    unsigned char* out = A.stream + at;
    if (A.layout) {
        const float4* src = reinterpret_cast<const float4*>(A.layout + (size_t)kSlabHeaderBytes * t + 2 * (size_t)e0);
        float4* head = reinterpret_cast<float4*>(out);
        float4* cols = reinterpret_cast<float4*>(out + kSlabHeaderBytes + 72 * ne);
        for (int i = threadIdx.x; i < kSlabHeaderBytes / 16 + ne / 8; i += kWideFillThreads)
            (i < kSlabHeaderBytes / 16 ? head[i] : cols[i - kSlabHeaderBytes / 16]) = __ldg(src + i);
        return;
    }
    double2* dst = reinterpret_cast<double2*>(out + kSlabHeaderBytes);
    for (int f2 = threadIdx.x; f2 < 9 * ne / 2; f2 += kWideFillThreads) {
        double v[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int f = 2 * f2 + q, e = f / 9, j = f - 9 * e;
            const unsigned s = __ldg(A.fill_src + e0 + e);
            const unsigned k = s & ~kSlabLowerBit;
            const int jj = (s & kSlabLowerBit) ? 3 * (j % 3) + j / 3 : j;
            v[q] = s != kSlabNoPos && k < (unsigned)A.nnz ? __ldg(A.values + 9 * (size_t)k + jj) : 0.0;
        }
        dst[f2] = make_double2(v[0], v[1]);
    }
}

}  // namespace

namespace {
template <class Real>
const void* part_kernel(bool float_sums)
{
    if constexpr (sizeof(Real) == 4)
        if (float_sums) return (const void*)pcg_part_kernel<Real, true>;
    return (const void*)pcg_part_kernel<Real, false>;
}
}  // namespace

template <class Real>
int pcg_part_max_grid()
{
    int dev = 0, sms = 0, per_sm = 1 << 20;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    for (const bool float_sums : {false, true}) {
        const void* k = part_kernel<Real>(float_sums);
        int b = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPartSmemLimit) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, kPartThreads, kPartSmemLimit) != cudaSuccess)
            return 0;
        per_sm = b < per_sm ? b : per_sm;
    }
    return sms * per_sm < kTagMaxGroup ? sms * per_sm : kTagMaxGroup;
}

template <class Real>
cudaError_t launch_pcg_part_kernel(const PartPcgArgs<Real>& args, int grid, cudaStream_t stream)
{
    PartPcgArgs<Real> a = args;
    void* kargs[] = {&a};
    const size_t smem = args.ring_offset + size_t(args.stages) * part_stage(sizeof(Real)) + part_table(sizeof(Real));
    const void* k = part_kernel<Real>(args.float_sums != 0);
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPartSmemLimit);
    if (e != cudaSuccess) return e;
    return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(kPartThreads), kargs, smem,
                                       stream);
}
template int pcg_part_max_grid<float>();
template int pcg_part_max_grid<double>();
template cudaError_t launch_pcg_part_kernel<float>(const PartPcgArgs<float>&, int, cudaStream_t);
template cudaError_t launch_pcg_part_kernel<double>(const PartPcgArgs<double>&, int, cudaStream_t);

cudaError_t launch_wide_fill_kernel(const WideFillArgs& args, cudaStream_t stream)
{
    if (args.tile_count <= 0) return cudaSuccess;
    wide_fill_kernel<<<args.tile_count, kWideFillThreads, 0, stream>>>(args);
    return cudaGetLastError();
}

}  // namespace pk
