// pk_selftest.cu -- the bounded waits of the PCG kernels made to run out on purpose.
//
// Every PCG kernel here waits for the other blocks of its group through the arrival
// counter of count_exchange (pk_device.cuh); each wait gives up after a number of polls,
// sets the error flag and lets the kernel leave through its normal exit, so a lost block
// costs a timeout status instead of a hung GPU.  This launch checks that path on the
// device: `blocks` co-resident blocks (one cooperative launch) exchange two partial sums
// as a group of `blocks + missing` members.  With missing = 0 every block gets the exact
// group sums; with missing > 0 the counter can never reach its target, every wait stops
// after `limit` polls and every block reports the timeout.  No counterpart in the
// reference (its solver runs on one CPU thread and never waits).
//
// The resident and the part-resident kernel wait for tagged packets instead.  Their exchange
// of sums runs here in the same way (tag_wait_selftest_kernel, with the wait for a
// shared-memory word beside it), and the kernels themselves on a small system one of whose
// parts sends none of its rows (pk_pcg_wait_selftest), so that the waits for rows -- the
// resident kernel's polls, its cluster's barrier phase, the part kernel's halo warp -- run out.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "../../../include/pkcuda.h"
#include "pk_device.cuh"
#include "pk_exchange.cuh"
#include "pk_res_plan.h"

namespace pk {
namespace {

__global__ void __launch_bounds__(128) exchange_wait_selftest_kernel(ExSlot* slots, unsigned* counter, GridSync* sync,
                                                                      int group, unsigned long long limit,
                                                                      double* out)
{
    __shared__ double sh[3 * 32];
    __shared__ int shi[32];
    // thread 0 holds the block's values (the exchange first sums over the block's threads)
    double v[2] = {threadIdx.x == 0 ? double(blockIdx.x + 1) : 0.0, threadIdx.x == 0 ? 1.0 : 0.0};
    int bad = 0;
    const bool ok = count_exchange<double, 2>(slots, counter, 0, group, sync, 1u, v, bad, sh, shi, limit);
    if (threadIdx.x == 0) {
        out[3 * blockIdx.x] = ok ? 1.0 : 0.0;
        out[3 * blockIdx.x + 1] = v[0];
        out[3 * blockIdx.x + 2] = v[1];
    }
}

// Four values per block: the exchange completed, its two sums, a word that nothing sets was seen.
constexpr int kTagTestThreads = 128;
__global__ void __launch_bounds__(kTagTestThreads)
    tag_wait_selftest_kernel(unsigned char* inbox, int members, unsigned* flags, unsigned limit, double* out)
{
    __shared__ TagShared sh;
    __shared__ int never;
    if (threadIdx.x == 0) {
        tag_init(sh);
        never = 0;
    }
    __syncthreads();
    double v[kTagSums] = {0.0, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0) {
        v[0] = double(blockIdx.x + 1);
        v[1] = 1.0;
    }
    unsigned bits = 0;
    const bool ok = tag_exchange(inbox, members, (int)blockIdx.x, 1u, v, bits, kTagTestThreads / 32, flags,
                                 TagTeam{kTagTestThreads / 32, 1}, sh, limit);
    const bool seen = wait_shared(&never, 1, limit);
    if (threadIdx.x == 0) {
        double* o = out + 4 * blockIdx.x;
        o[0] = ok ? 1.0 : 0.0;
        o[1] = v[0];
        o[2] = v[1];
        o[3] = seen ? 1.0 : 0.0;
    }
}

// Device copies of host arrays, freed together.
struct Arena {
    std::vector<void*> held;
    bool ok = true;
    void* raw(const void* src, size_t bytes)  // src NULL: zeros
    {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes + 1024) != cudaSuccess) {
            ok = false;
            return nullptr;
        }
        held.push_back(p);
        const cudaError_t e =
            src ? cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice) : cudaMemset(p, 0, bytes + 1024);
        ok = ok && e == cudaSuccess;
        return p;
    }
    template <class D, class T>
    D* up(const std::vector<T>& v)
    {
        return static_cast<D*>(raw(v.data(), v.size() * sizeof(T)));
    }
    template <class D>
    D* zeros(size_t bytes)
    {
        return static_cast<D*>(raw(nullptr, bytes));
    }
    ~Arena()
    {
        for (void* p : held) cudaFree(p);
    }
};

}  // namespace
}  // namespace pk

extern "C" PKCUDA_API int pk_tag_wait_selftest(int device, int blocks, int missing, unsigned limit, double* out)
{
    if (blocks < 2 || blocks > 64 || missing < 0 || missing > 64 || !out || limit == 0) return PK_ERR_ARG;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return PK_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return PK_ERR_CUDA;
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk::tag_wait_selftest_kernel, pk::kTagTestThreads, 0) !=
            cudaSuccess ||
        blocks > sms * per_sm)
        return PK_ERR_UNSUPPORTED;
    pk::Arena mem;
    int members = blocks + missing;
    unsigned char* inbox =
        mem.zeros<unsigned char>(2 * static_cast<size_t>(members) * members * pk::kTagSlotBytes);
    unsigned* flags = mem.zeros<unsigned>(sizeof(unsigned));
    double* d_out = mem.zeros<double>(4 * sizeof(double) * blocks);
    if (!mem.ok) return PK_ERR_CUDA;
    void* args[] = {&inbox, &members, &flags, &limit, &d_out};
    unsigned fl = 0;
    if (cudaLaunchCooperativeKernel((const void*)pk::tag_wait_selftest_kernel, dim3(blocks), dim3(pk::kTagTestThreads),
                                    args, 0, nullptr) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(out, d_out, 4 * sizeof(double) * blocks, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(&fl, flags, sizeof(fl), cudaMemcpyDeviceToHost) != cudaSuccess)
        return PK_ERR_CUDA;
    return (fl & pk::kFlagBarrierTimeout) ? PK_ERR_TIMEOUT : PK_OK;
}

// A band of 700 rows in FP64 (20 on the diagonal, -1 towards the next five rows) on four blocks.
extern "C" PKCUDA_API int pk_pcg_wait_selftest(int device, int kernel, int lost, unsigned limit, double* x,
                                               int* iterations)
{
    constexpr int n = 700, band = 6, parts = 4;
    if (kernel < 0 || kernel > 2 || limit == 0 || !x || !iterations) return PK_ERR_ARG;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return PK_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return PK_ERR_CUDA;
    std::vector<int> rs(1, 0), col;
    std::vector<double> values, b(3 * n), minv(9 * n, 0.0), coords(3 * n, 0.0);
    for (int r = 0; r < n; ++r) {
        for (int c = r; c < n && c < r + band; ++c) {
            col.push_back(c);
            for (int e = 0; e < 9; ++e) values.push_back(e % 4 ? 0.0 : c == r ? 20.0 : -1.0);
        }
        rs.push_back(static_cast<int>(col.size()));
        coords[3 * r] = r;
        for (int a = 0; a < 3; ++a) {
            b[3 * r + a] = std::sin(3.0 * r + a);
            minv[9 * r + 4 * a] = 0.05;
        }
    }
    const int nnz = rs[n];
    std::vector<int> lts(n + 1), ltr(nnz - n), ltb(nnz - n);
    const int lower = pk_bsr_transpose_index(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data());
    if (lower < 0) return lower;
    pk::Arena mem;
    pk::DevStats* st = mem.zeros<pk::DevStats>(sizeof(pk::DevStats));
    double* d_x = mem.zeros<double>(3 * n * sizeof(double));
    cudaError_t e = cudaSuccess;
    if (kernel < 2) {
        pk::ResLimits limits;
        limits.blocks = parts;
        if (kernel == 1) limits.clusters[2] = 1;
        if (pk::pcg_res_limits<double>().blocks < parts) return PK_ERR_UNSUPPORTED;
        const int seg[2] = {0, n};
        pk::ResPlan plan;
        if (!pk::build_res_plan(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data(), coords.data(), seg, 1,
                                limits, 8, plan).empty() ||
            (plan.cluster > 0) != (kernel == 1) || plan.max_group < 2)
            return PK_ERR_UNSUPPORTED;
        if (lost) plan.part_info[10] = 0;
        pk::ResPcgArgs<double> a{};
        a.n = n;
        a.lpr = plan.lpr;
        a.nslots = plan.slots;
        a.tmem_slots = plan.tmem;
        a.max_halo = plan.max_halo;
        a.part_info = mem.up<int>(plan.part_info);
        a.perm = mem.up<int>(plan.perm);
        a.halo_src = mem.up<int>(plan.halo_src);
        a.halo_count = static_cast<int>(plan.halo_src.size());
        a.send = mem.up<int2>(plan.send);
        a.src = mem.up<unsigned>(plan.src);
        a.col = mem.up<unsigned short>(plan.col);
        a.slot_count = plan.slots * plan.parts;
        a.nnz = nnz;
        a.smem_bytes = static_cast<unsigned>(plan.smem_bytes);
        a.values = mem.up<double>(values);
        a.b = mem.up<double>(b);
        a.minv = mem.up<double>(minv);
        a.x = d_x;
        a.rows_in = mem.zeros<unsigned char>(2 * plan.halo_src.size() * pk::res_row_packet(8));
        a.sums_in = mem.zeros<unsigned char>(2 * static_cast<size_t>(plan.parts) * plan.max_group * pk::kResSlotBytes);
        a.sums_stride = static_cast<size_t>(plan.max_group) * pk::kResSlotBytes;
        a.epoch = mem.zeros<unsigned>(sizeof(unsigned) * plan.parts);
        a.spin_limit = limit;
        a.max_iterations = 100;
        a.tolerance = 1e-10;
        a.flags = &st->flags;
        a.stats = st;
        a.nbodies = 1;
        if (!mem.ok) return PK_ERR_CUDA;
        e = pk::launch_pcg_res_kernel<double>(a, plan.threads, plan.rpt, plan.cluster, plan.parts, nullptr);
    } else {
        if (pk::pcg_part_max_grid<double>() < parts) return PK_ERR_UNSUPPORTED;
        pk::SlabPlan plan;
        if (!pk::build_slab_plan(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data(), coords.data(), parts,
                                 plan, pk::kSlabFull, true).empty())
            return PK_ERR_UNSUPPORTED;
        if (lost) plan.send_start[0] = plan.send_start[1];
        const int halo = static_cast<int>(plan.halo_src.size());
        pk::PartPcgArgs<double> a{};
        a.n = n;
        a.part_info = mem.up<int>(plan.part_info);
        a.send_start = mem.up<int>(plan.send_start);
        a.send = mem.up<int2>(plan.send);
        a.tile_desc = mem.up<int4>(plan.tile_desc);
        a.tile_count = static_cast<int>(plan.tile_desc.size() / 4);
        a.halo_count = halo;
        unsigned char* stream = mem.zeros<unsigned char>(plan.stream_bytes);
        a.stream = stream;
        a.stream_bytes = plan.stream_bytes;
        a.win_cap = plan.max_window;
        a.stages = pk::part_stages(8, a.win_cap);
        a.ring_offset = static_cast<unsigned>(pk::part_ring_offset(8, a.win_cap));
        a.spin_limit = limit;
        a.rows_in = mem.zeros<unsigned char>(32 * static_cast<size_t>(halo) +
                                             2 * pk::kResSlotBytes * static_cast<size_t>(plan.parts) * plan.parts);
        a.sums_in = a.rows_in + 32 * static_cast<size_t>(halo);
        a.perm = mem.up<int>(plan.perm);
        a.b = mem.up<double>(b);
        a.minv = mem.up<double>(minv);
        a.x = d_x;
        a.qs = mem.zeros<double>(4 * n * sizeof(double));
        a.mrow = mem.zeros<double>(9 * n * sizeof(double));
        a.max_iterations = 100;
        a.tolerance = 1e-10;
        a.flags = &st->flags;
        a.stats = st;
        pk::WideFillArgs f{};
        f.values = mem.up<double>(values);
        f.nnz = nnz;
        f.tile_desc = a.tile_desc;
        f.tile_entry0 = mem.up<int>(plan.tile_entry0);
        f.tile_count = a.tile_count;
        f.entries = static_cast<int>(plan.fill_src.size());
        f.fill_src = mem.up<unsigned>(plan.fill_src);
        f.stream = stream;
        f.stream_bytes = plan.stream_bytes;
        f.layout = mem.up<unsigned char>(plan.stream);
        if (!mem.ok) return PK_ERR_CUDA;
        e = pk::launch_wide_fill_kernel(f, nullptr);
        f.layout = nullptr;
        if (e == cudaSuccess) e = pk::launch_wide_fill_kernel(f, nullptr);
        if (e == cudaSuccess) e = pk::launch_pcg_part_kernel<double>(a, plan.parts, nullptr);
    }
    pk::DevStats out{};
    if (e != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(&out, st, sizeof(out), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(x, d_x, 3 * n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return PK_ERR_CUDA;
    *iterations = out.iterations;
    if (out.flags & pk::kFlagBarrierTimeout) return PK_ERR_TIMEOUT;
    return (out.flags & pk::kFlagConverged) ? PK_OK : PK_ERR_STATE;
}

extern "C" PKCUDA_API int pk_exchange_wait_selftest(int device, int blocks, int missing, unsigned long long limit,
                                                    double* out)
{
    if (blocks < 2 || blocks > 64 || missing < 0 || missing > 64 || !out || limit == 0) return PK_ERR_ARG;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return PK_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return PK_ERR_CUDA;
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk::exchange_wait_selftest_kernel, 128, 0) !=
            cudaSuccess ||
        blocks > sms * per_sm)
        return PK_ERR_UNSUPPORTED;
    // Slots for both generation buffers of the larger of the grid and the group, the
    // counter and the sync word, the per-block results.
    const int members = blocks + missing;
    const size_t slot_bytes = 2 * sizeof(pk::ExSlot) * static_cast<size_t>(members);
    const size_t out_bytes = 3 * sizeof(double) * static_cast<size_t>(blocks);
    unsigned char* mem = nullptr;
    const size_t total = slot_bytes + 256 + out_bytes;
    if (cudaMalloc(&mem, total) != cudaSuccess) return PK_ERR_CUDA;
    int rc = PK_OK;
    pk::ExSlot* slots = reinterpret_cast<pk::ExSlot*>(mem);
    unsigned* counter = reinterpret_cast<unsigned*>(mem + slot_bytes);
    pk::GridSync* sync = reinterpret_cast<pk::GridSync*>(mem + slot_bytes + 128);
    double* d_out = reinterpret_cast<double*>(mem + slot_bytes + 256);
    if (cudaMemset(mem, 0, total) != cudaSuccess) rc = PK_ERR_CUDA;
    if (rc == PK_OK) {
        int group = members;
        void* args[] = {&slots, &counter, &sync, &group, &limit, &d_out};
        if (cudaLaunchCooperativeKernel((const void*)pk::exchange_wait_selftest_kernel, dim3(blocks), dim3(128), args,
                                        0, nullptr) != cudaSuccess ||
            cudaDeviceSynchronize() != cudaSuccess)
            rc = PK_ERR_CUDA;
    }
    if (rc == PK_OK && cudaMemcpy(out, d_out, out_bytes, cudaMemcpyDeviceToHost) != cudaSuccess) rc = PK_ERR_CUDA;
    int err = 0;
    if (rc == PK_OK && cudaMemcpy(&err, &sync->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = PK_ERR_CUDA;
    cudaFree(mem);
    if (rc == PK_OK && err) rc = PK_ERR_TIMEOUT;
    return rc;
}
