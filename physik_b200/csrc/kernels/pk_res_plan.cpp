// pk_res_plan.cpp -- builds the resident PCG kernel's layout (see pk_res_plan.h).
#include "pk_res_plan.h"

#include <algorithm>
#include <atomic>
#include <new>
#include <numeric>

#include "pk_slab_plan.h"

namespace pk {
namespace {

// Cycles of one iteration, fitted to measurements on B200 (1.93 GHz).  A block's own work:
// 2,580 with 44 FP32 rows, 3,100 with 125, 3,900 with 164 (one lane per row: fewer loads in
// flight); 3,300 with 32 FP64 rows, 4,670 with 125.  An exchange: none for one block, 500 to 900 in clusters of 4 to 16, 1,900 to
// 3,300 among 41 to 148 blocks through global memory.
double block_cycles(int rows, int real, int lpr)
{
    return (real == 4 ? 2000.0 + 9.0 * rows : 2800.0 + 16.0 * rows) + (lpr == 1 ? 500.0 : 0.0);
}
double exchange_cycles(int group, bool cluster)
{
    if (group <= 1) return 0.0;
    return cluster ? 420.0 + 30.0 * group : 1500.0 + 12.0 * group;
}

// How the launch is cut: rows per part aimed at, the cluster size (0: global exchange) and
// the threads of a block at most.
struct Cut {
    int per, cluster, cap;
    double cycles;
    bool pairs = false;  // two rows a thread
};

// Lanes per row, the most that keep the block under its threads, and the threads.
struct Lanes {
    int lpr, threads;
};
Lanes lanes_for(int rows, int cap)
{
    Lanes l{8, 0};
    for (;; l.lpr /= 2) {
        l.threads = std::max(kResMinThreads, (rows * l.lpr + 31) / 32 * 32);
        if (l.threads <= cap || l.lpr == 1) return l;
    }
}

// Recursive coordinate bisection of ids[lo, hi) into parts of equal rows: split across the
// widest axis (ties by row), so the result depends only on the inputs.
void bisect(int* ids, int lo, int hi, int part0, int parts, const double* xyz, int* part_of)
{
    if (parts <= 1) {
        for (int i = lo; i < hi; ++i) part_of[ids[i]] = part0;
        return;
    }
    double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
    for (int i = lo; i < hi; ++i)
        for (int a = 0; a < 3; ++a) {
            mn[a] = std::min(mn[a], xyz[3 * (size_t)ids[i] + a]);
            mx[a] = std::max(mx[a], xyz[3 * (size_t)ids[i] + a]);
        }
    int ax = 0;
    for (int a = 1; a < 3; ++a)
        if (mx[a] - mn[a] > mx[ax] - mn[ax]) ax = a;
    const int left = parts / 2, cut = lo + static_cast<int>(((long long)(hi - lo) * left + parts / 2) / parts);
    std::nth_element(ids + lo, ids + cut, ids + hi, [&](int a, int b) {
        const double ca = xyz[3 * (size_t)a + ax], cb = xyz[3 * (size_t)b + ax];
        return ca < cb || (ca == cb && a < b);
    });
    bisect(ids, lo, cut, part0, left, xyz, part_of);
    bisect(ids, cut, hi, part0 + left, parts - left, xyz, part_of);
}

int parts_of(int rows, int per) { return rows <= 0 ? 0 : (rows + per - 1) / per; }

// Groups of the bodies in clusters of c blocks, largest first into the first cluster with
// room; place[b] = first block.  Returns the clusters used.
int pack(const std::vector<int>& group, int c, std::vector<int>& place)
{
    std::vector<int> order(group.size()), fill;
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return group[a] > group[b]; });
    place.assign(group.size(), -1);
    size_t open = 0;
    for (const int b : order) {
        if (group[b] == 0) continue;
        size_t k = open;
        while (k < fill.size() && fill[k] + group[b] > c) ++k;
        if (k == fill.size()) fill.push_back(0);
        place[b] = static_cast<int>(k) * c + fill[k];
        fill[k] += group[b];
        while (open < fill.size() && fill[open] == c) ++open;
    }
    return static_cast<int>(fill.size());
}

std::string build_cut(int n, const int* row_start, const int* col, const int* lt_start, const int* lt_row,
                      const int* lt_block, const double* coords, const int* seg, int nseg, const std::vector<int>& len,
                      const Cut& cut, int max_blocks, int real, ResPlan& out)
{
    out = ResPlan{};
    // 1. parts of the bodies and their places
    std::vector<int> group(nseg), place;
    for (int b = 0; b < nseg; ++b) group[b] = parts_of(seg[b + 1] - seg[b], cut.per);
    int parts;
    if (cut.cluster > 0) {
        for (int b = 0; b < nseg; ++b)
            if (group[b] > cut.cluster) return "a body exceeds a cluster";
        parts = pack(group, cut.cluster, place) * cut.cluster;
    } else {
        place.assign(nseg, 0);
        parts = 0;
        for (int b = 0; b < nseg; ++b) {
            place[b] = parts;
            parts += group[b];
        }
        if (parts > max_blocks) return "more parts than blocks";
    }
    std::vector<int> part_of(n, 0), body(parts, 0), gfirst(parts, 0), gsize(parts, 0), rows_of(parts, 0);
    {
        std::vector<int> ids(n);
        std::iota(ids.begin(), ids.end(), 0);
        for (int b = 0; b < nseg; ++b) {
            const int k = group[b];
            if (k == 0) continue;
            bisect(ids.data(), seg[b], seg[b + 1], place[b], k, coords, part_of.data());
            for (int r = seg[b]; r < seg[b + 1]; ++r)
                out.max_rows = std::max(out.max_rows, ++rows_of[part_of[r]]);
            for (int p = place[b]; p < place[b] + k; ++p) {
                if (rows_of[p] == 0) return "a part has no rows";
                body[p] = b;
                gfirst[p] = place[b];
                gsize[p] = k;
            }
            out.max_group = std::max(out.max_group, k);
        }
    }
    // 2. lanes
    const Lanes lanes = cut.pairs ? Lanes{1, std::max(kResMinThreads, (out.max_rows + 63) / 64 * 32)}
                                  : lanes_for(out.max_rows, cut.cap);
    if (lanes.threads > (cut.pairs ? kResPairThreads : kResMaxThreads)) return "a part has more rows than threads";
    out.lpr = lanes.lpr;
    out.threads = lanes.threads;
    out.rpt = cut.pairs ? 2 : 1;
    out.real = real;
    out.n = n;
    out.parts = parts;
    out.cluster = cut.cluster;
    const int T = out.threads;
    for (int r = 0; r < n; ++r) out.slots = std::max(out.slots, (len[r] + out.lpr - 1) / out.lpr);
    out.slots *= out.rpt;
    // 3. part order: parts in order, rows ascending
    std::vector<int> start(parts + 1, 0), inv(n);
    for (int p = 0; p < parts; ++p) start[p + 1] = start[p] + rows_of[p];
    out.perm.resize(n);
    {
        std::vector<int> fill(start.begin(), start.end() - 1);
        for (int r = 0; r < n; ++r) {
            inv[r] = fill[part_of[r]]++;
            out.perm[inv[r]] = r;
        }
    }
    // 4. halos
    std::atomic<bool> failed{false};
    auto each_part = [&](const std::function<void(int, int)>& f) {
        const auto guarded = [&](int p, int t) {
            try {
                f(p, t);
            } catch (...) {  // nothing may leave a worker thread
                failed = true;
            }
        };
        if (n >= 4096)
            for_items(parts, guarded);
        else
            for (int p = 0; p < parts; ++p) guarded(p, 0);
    };
    std::vector<std::vector<int>> halos(parts);
    each_part([&](int p, int) {
        std::vector<int>& halo = halos[p];
        for (int g = start[p]; g < start[p + 1]; ++g) {
            const int r = out.perm[g];
            for (int k = row_start[r]; k < row_start[r + 1]; ++k)
                if (part_of[col[k]] != p) halo.push_back(inv[col[k]]);
            for (int e = lt_start[r]; e < lt_start[r + 1]; ++e)
                if (part_of[lt_row[e]] != p) halo.push_back(inv[lt_row[e]]);
        }
        std::sort(halo.begin(), halo.end());
        halo.erase(std::unique(halo.begin(), halo.end()), halo.end());
    });
    if (failed) return kNoMemory;
    out.part_info.assign((size_t)kResPartInts * parts, 0);
    for (int p = 0; p < parts; ++p) {
        int* pi = out.part_info.data() + (size_t)kResPartInts * p;
        const std::vector<int>& halo = halos[p];
        for (const int g : halo)
            if (gsize[p] <= 1 || gfirst[part_of[out.perm[g]]] != gfirst[p]) return "a block couples two bodies";
        const int m = rows_of[p], h = static_cast<int>(halo.size());
        if (h > res_halo_per_thread(out.rpt) * T) return "a part's halo exceeds its threads";
        if (3 * (m + h) > 65535) return "a part's window exceeds its column index";
        pi[0] = start[p];
        pi[1] = m;
        pi[2] = static_cast<int>(out.halo_src.size());
        pi[3] = h;
        pi[4] = out.slots * p;
        pi[6] = gfirst[p];
        pi[7] = gsize[p];
        pi[8] = body[p];
        out.max_halo = std::max(out.max_halo, h);
        out.halo_src.insert(out.halo_src.end(), halo.begin(), halo.end());
    }
    // Tensor memory takes as many slots as it holds where a thread has two rows, and in FP64
    // where shared memory is too small (the path costs 2 % where it is not): blocks that may share an SM (half its
    // shared memory each) must not ask for it.
    const auto most_bytes = [&] {
        size_t most = 0;
        for (int p = 0; p < parts; ++p)
            most = std::max(most, res_smem_bytes(real, T, rows_of[p], out.part_info[(size_t)kResPartInts * p + 3],
                                                 out.smem_slots(), out.tmem, out.cluster, out.max_halo));
        return most;
    };
    const int batch = res_tmem_batch(real), in_regs = res_reg_slots(real, T, out.rpt);
    const int fit = std::min(res_tmem_slots(real, T), (std::max(0, out.slots - in_regs) + batch - 1) / batch * batch);
    if (cut.pairs) out.tmem = fit;
    out.smem_bytes = most_bytes();
    if (out.smem_bytes > kResSmemLimit && real == 8 && cut.cluster == 0 && T <= 256) {
        out.tmem = fit;
        out.smem_bytes = most_bytes();
    }
    if (out.tmem > 0) out.smem_bytes = std::max(out.smem_bytes, kResAloneBytes);
    if (out.smem_bytes > kResSmemLimit) return "a part's rows exceed on-chip memory";
    if ((size_t)out.slots * parts * T > 0x7fffffffull) return "too many slots";
    // 5. slots
    struct Entry {
        int win;
        unsigned src;
    };
    out.src.assign((size_t)out.slots * parts * T, kSlabNoPos);
    out.col.assign((size_t)out.slots * parts * T, 0);
    std::vector<std::vector<int>> scratch(n >= 4096 ? plan_thread_count() : 1);
    each_part([&](int p, int t) {
        std::vector<int>& win = scratch[t];
        win.resize(n);  // only the entries set below are read
        std::vector<Entry> row;
        const int* pi = out.part_info.data() + (size_t)kResPartInts * p;
        const int g0 = pi[0], m = pi[1], h = pi[3];
        for (int i = 0; i < m; ++i) win[out.perm[g0 + i]] = i;
        for (int i = 0; i < h; ++i) win[out.perm[out.halo_src[pi[2] + i]]] = m + i;
        for (int i = 0; i < m; ++i) {
            const int r = out.perm[g0 + i];
            row.clear();
            for (int k = row_start[r]; k < row_start[r + 1]; ++k)
                row.push_back({win[col[k]], static_cast<unsigned>(k)});
            for (int e = lt_start[r]; e < lt_start[r + 1]; ++e)
                row.push_back({win[lt_row[e]], static_cast<unsigned>(lt_block[e]) | kSlabLowerBit});
            std::sort(row.begin(), row.end(), [](const Entry& a, const Entry& b) { return a.win < b.win; });
            for (size_t j = 0; j < row.size(); ++j) {
                const size_t at = out.rpt == 1
                                      ? ((size_t)pi[4] + j / out.lpr) * T + (size_t)i * out.lpr + j % out.lpr
                                      : ((size_t)pi[4] + 2 * j + i / T) * T + i % T;
                out.src[at] = row[j].src;
                out.col[at] = static_cast<unsigned short>(3 * row[j].win);
            }
        }
    });
    if (failed) return kNoMemory;
    // 6. who sends which row where
    std::vector<std::vector<int>> sends(parts);
    for (int p = 0; p < parts; ++p) {
        const int* pi = out.part_info.data() + (size_t)kResPartInts * p;
        for (int i = 0; i < pi[3]; ++i) {
            const int g = out.halo_src[pi[2] + i], q = part_of[out.perm[g]];
            sends[q].push_back(g - start[q]);
            sends[q].push_back(out.cluster > 0 ? ((p % out.cluster) << 16) | i : pi[2] + i);
        }
    }
    for (int p = 0; p < parts; ++p) {
        int* pi = out.part_info.data() + (size_t)kResPartInts * p;
        pi[9] = static_cast<int>(out.send.size() / 2);
        pi[10] = static_cast<int>(sends[p].size() / 2);
        out.send.insert(out.send.end(), sends[p].begin(), sends[p].end());
    }
    return "";
}

}  // namespace

std::string build_res_plan(int n, const int* row_start, const int* col, const int* lt_start, const int* lt_row,
                           const int* lt_block, const double* coords, const int* seg, int nseg,
                           const ResLimits& limits, int real, ResPlan& out)
try {
    out = ResPlan{};
    if (n <= 0 || nseg <= 0 || limits.blocks <= 0 || seg[0] != 0 || seg[nseg] != n) return "empty system";
    std::vector<double> held;
    coords = finite_coords(n, coords, held);
    std::vector<int> len(n);
    int longest = 0, largest = 0;
    for (int r = 0; r < n; ++r) {
        len[r] = (row_start[r + 1] - row_start[r]) + (lt_start[r + 1] - lt_start[r]);
        longest = std::max(longest, len[r]);
    }
    for (int b = 0; b < nseg; ++b) largest = std::max(largest, seg[b + 1] - seg[b]);
    // Candidate cuts, fastest estimate first; the first that fits is taken.  Blocks of at
    // most 256 threads: every warp pays the exchange's and the scalars' instructions, and
    // 512 threads measured 25 to 50 % slower per iteration at every size tried.  A cluster
    // launch of more clusters than are resident runs in waves; blocks of 128 threads and
    // half the shared memory run two to an SM, each about 1.4 times slower.
    std::vector<Cut> cuts;
    const int max_blocks = std::min(limits.blocks, kResMaxParts);
    std::vector<int> group(nseg), place;
    std::vector<int> pers;
    for (int per = 16; per <= 2 * kResPairThreads; per += per < 64 ? 4 : 8) pers.push_back(per);
    for (int q = 0; q < 5; ++q) {
        const int c = 1 << q;
        if (limits.clusters[q] <= 0) continue;
        for (const int per : pers) {
            if (parts_of(largest, per) > c || per > kResMaxThreads) continue;
            if (c > 1 && parts_of(largest, per) <= c / 2) break;  // a smaller cluster does it
            for (int b = 0; b < nseg; ++b) group[b] = parts_of(seg[b + 1] - seg[b], per);
            const int waves = (pack(group, c, place) + limits.clusters[q] - 1) / limits.clusters[q];
            const int rows = std::min(largest, per);
            const int cap = rows > 256 ? 512 : 256;
            cuts.push_back(
                {per, c, cap, waves * (block_cycles(rows, real, lanes_for(rows, cap).lpr) + exchange_cycles(c, true))});
            const Lanes l = lanes_for(rows, 128);
            const int slots = std::max(0, (longest + l.lpr - 1) / l.lpr - res_reg_slots(real, l.threads, 1));
            if (waves > 1 && l.threads == 128 && slots * 128 * (9 * real + 2) < 80 * 1024)
                cuts.push_back({per, c, 128,
                                (waves + 1) / 2 * 1.4 * (block_cycles(rows, real, l.lpr) + exchange_cycles(c, true))});
        }
    }
    for (const int per : pers) {
        long long total = 0;
        for (int b = 0; b < nseg; ++b) total += parts_of(seg[b + 1] - seg[b], per);
        if (total > max_blocks) continue;
        const int k = parts_of(largest, per);
        const int rows = std::min(largest, per);
        // More rows than 256 threads: two a thread in FP32 (16 warps pay the exchange and the
        // sums more than 10 pay a second row).
        const bool pairs = real == 4 && rows > 256;
        if (!pairs && rows > kResMaxThreads) continue;
        const int cap = rows > 256 ? 512 : 256;
        cuts.push_back({per, 0, cap,
                        block_cycles(rows, real, pairs ? 1 : lanes_for(rows, cap).lpr) + exchange_cycles(k, false),
                        pairs});
    }
    if (cuts.empty()) return "more rows than the blocks hold";
    std::stable_sort(cuts.begin(), cuts.end(), [](const Cut& a, const Cut& b) { return a.cycles < b.cycles; });
    std::string why;
    for (const Cut& c : cuts) {
        // memory of the values alone, before a layout is built
        const double rows = std::min<double>(c.per, largest);
        const int T = c.pairs ? std::max(kResMinThreads, ((int)rows + 63) / 64 * 32) : lanes_for((int)rows, c.cap).threads;
        const double off_smem = 9.0 * real * T *
                                (res_reg_slots(real, T, c.pairs ? 2 : 1) +
                                 (c.pairs || (real == 8 && c.cluster == 0 && T <= 256) ? res_tmem_slots(real, T) : 0));
        if (rows * longest * (9 * real + 2) - off_smem > 1.0 * kResSmemLimit) continue;
        why = build_cut(n, row_start, col, lt_start, lt_row, lt_block, coords, seg, nseg, len, c, max_blocks, real, out);
        if (why.empty()) return why;
    }
    return why.empty() ? "a part's rows exceed on-chip memory" : why;
} catch (const std::bad_alloc&) {
    return kNoMemory;
}

std::string res_check(const ResPlan& plan, int nnz, const ResLimits& limits, int real)
{
    if (plan.parts < 1) return "no parts";
    if (plan.cluster == 0 ? plan.parts > limits.blocks || plan.max_group > kResMaxParts
                          : plan.cluster > kResMaxCluster || plan.parts % plan.cluster != 0)
        return "bad part count";
    if (plan.lpr != 1 && plan.lpr != 2 && plan.lpr != 4 && plan.lpr != 8) return "bad lanes per row";
    const int T = plan.threads;
    if (T < kResMinThreads || T > (plan.rpt == 2 ? kResPairThreads : kResMaxThreads) || T % 32 != 0)
        return "bad threads";
    if (plan.rpt != 1 && (plan.rpt != 2 || plan.lpr != 1 || plan.cluster != 0 || real != 4)) return "bad rows per thread";
    if (plan.slots % plan.rpt != 0) return "bad slots";
    if (plan.tmem < 0 || plan.tmem % res_tmem_batch(real) != 0 || plan.tmem > res_tmem_slots(real, T) ||
        (plan.tmem > 0 && (plan.smem_bytes < kResAloneBytes || plan.cluster != 0)))
        return "bad tensor memory";
    if (plan.smem_bytes > kResSmemLimit) return "too much shared memory";
    const size_t slot_count = plan.src.size() / T;
    if (plan.send.size() != 2 * plan.halo_src.size()) return "bad send lists";
    std::vector<int> part_of(plan.n, -1);
    std::vector<unsigned char> owned(plan.n, 0), seen(nnz, 0);
    for (int p = 0; p < plan.parts; ++p) {
        const int* pi = plan.part_info.data() + (size_t)kResPartInts * p;
        if (pi[1] < (pi[7] > 0 ? 1 : 0) || pi[0] < 0 || pi[0] + pi[1] > plan.n || pi[1] * plan.lpr > T * plan.rpt)
            return "bad rows";
        if (pi[7] == 0 && pi[1] != 0) return "rows without a group";
        for (int g = pi[0]; g < pi[0] + pi[1]; ++g) {
            if (plan.perm[g] < 0 || plan.perm[g] >= plan.n || owned[plan.perm[g]]++) return "a row owned twice";
            part_of[g] = p;
        }
    }
    for (int p = 0; p < plan.parts; ++p) {
        const int* pi = plan.part_info.data() + (size_t)kResPartInts * p;
        const int m = pi[1], h = pi[3];
        if (pi[7] == 0) continue;
        if (h < 0 || h > res_halo_per_thread(plan.rpt) * T || h > plan.max_halo || pi[2] < 0 ||
            (size_t)pi[2] + h > plan.halo_src.size())
            return "bad halo";
        if (pi[4] < 0 || (size_t)pi[4] + plan.slots > slot_count) return "bad slots";
        if (pi[9] < 0 || pi[10] < 0 || (size_t)pi[9] + pi[10] > plan.halo_src.size()) return "bad sends";
        if (res_smem_bytes(real, T, m, h, plan.smem_slots(), plan.tmem, plan.cluster, plan.max_halo) > plan.smem_bytes) return "bad size";
        if (pi[7] > plan.max_group || pi[6] < 0 || p < pi[6] || p >= pi[6] + pi[7] || pi[6] + pi[7] > plan.parts)
            return "bad group";
        if (plan.cluster > 0 && pi[6] / plan.cluster != (pi[6] + pi[7] - 1) / plan.cluster)
            return "a group across clusters";
        for (int q = pi[6]; q < pi[6] + pi[7]; ++q) {
            const int* qi = plan.part_info.data() + (size_t)kResPartInts * q;
            if (qi[6] != pi[6] || qi[7] != pi[7] || qi[8] != pi[8]) return "mixed group";
        }
        for (int i = 0; i < h; ++i) {
            const int g = plan.halo_src[pi[2] + i];
            if (g < 0 || g >= plan.n || part_of[g] == p || part_of[g] < pi[6] || part_of[g] >= pi[6] + pi[7])
                return "a halo row outside the group";
            const int* qi = plan.part_info.data() + (size_t)kResPartInts * part_of[g];
            const int want = plan.cluster > 0 ? ((p % plan.cluster) << 16) | i : pi[2] + i;
            int found = 0;
            for (int e = qi[9]; e < qi[9] + qi[10]; ++e)
                found += plan.send[2 * (size_t)e] == g - qi[0] && plan.send[2 * (size_t)e + 1] == want;
            if (found != 1) return "a halo row nobody sends";
        }
        for (size_t at = (size_t)pi[4] * T; at < (size_t)(pi[4] + plan.slots) * T; ++at) {
            const unsigned s = plan.src[at];
            if (s == kSlabNoPos) continue;
            const unsigned k = s & ~kSlabLowerBit, bit = (s & kSlabLowerBit) ? 2u : 1u;
            if (k >= (unsigned)nnz || (seen[k] & bit)) return "a block placed twice";
            seen[k] |= bit;
            if (plan.col[at] % 3 != 0 || plan.col[at] + 2 >= 3 * (m + h)) return "a column outside the window";
        }
    }
    for (int r = 0; r < plan.n; ++r)
        if (!owned[r]) return "a row without an owner";
    for (int k = 0; k < nnz; ++k)
        if (!(seen[k] & 1)) return "a block not placed";
    return "";
}

void res_spmv_host(const ResPlan& plan, const double* values, const double* x, double* y)
{
    for (int p = 0; p < plan.parts; ++p) {
        const int* pi = plan.part_info.data() + (size_t)kResPartInts * p;
        const int m = pi[1], h = pi[3];
        std::vector<double> win(3 * (size_t)(m + h));
        for (int i = 0; i < m + h; ++i) {
            const int g = i < m ? pi[0] + i : plan.halo_src[pi[2] + i - m];
            for (int a = 0; a < 3; ++a) win[3 * (size_t)i + a] = x[3 * (size_t)plan.perm[g] + a];
        }
        for (int i = 0; i < m; ++i)
            for (int a = 0; a < 3; ++a) y[3 * (size_t)plan.perm[pi[0] + i] + a] = 0.0;
        for (int k = 0; k < plan.slots; ++k)
            for (int t = 0; t < plan.threads; ++t) {
                const int row = plan.rpt == 1 ? t / plan.lpr : t + k % 2 * plan.threads;
                if (row >= m) continue;
                const size_t at = ((size_t)pi[4] + k) * plan.threads + t;
                const unsigned s = plan.src[at];
                if (s == kSlabNoPos) continue;
                const double* v = values + 9 * (size_t)(s & ~kSlabLowerBit);
                const double* d = win.data() + plan.col[at];
                double* out = y + 3 * (size_t)plan.perm[pi[0] + row];
                for (int a = 0; a < 3; ++a)
                    for (int c = 0; c < 3; ++c) out[a] += v[(s & kSlabLowerBit) ? 3 * a + c : 3 * c + a] * d[c];
            }
    }
}

}  // namespace pk
