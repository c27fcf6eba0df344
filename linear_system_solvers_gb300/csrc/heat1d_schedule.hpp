// heat1d_schedule.hpp -- placement of the 1-D groups on the warps of a one-CTA-per-SM launch.
//
// A group (32 equal-size instances, one warp) runs its whole time loop in one warp, and group
// costs differ by up to ~40x in a batch of uneven instances.  With one group per warp in
// blockIdx order the SMs that receive the costliest groups finish long after the others.  The
// factorised sweep launches one CTA per SM instead, and this placement balances the work of
// every SM sub-partition (warp w of a CTA runs on sub-partition w % 4): groups go, costliest
// first, to the least-loaded (SM, sub-partition) bin -- ties to the lowest bin, numbered
// sub-partition-major so that the first groups spread over all SMs -- and a bin's groups go,
// costliest first, to the least-loaded of its warps.  A warp runs its groups one after the other.
// Host-only (no CUDA): the CPU tests compile it directly.
#pragma once

#include <algorithm>
#include <cmath>
#include <functional>
#include <numeric>
#include <queue>
#include <utility>
#include <vector>

namespace lss_gb300 {
namespace heat1d {

constexpr int SUBPARTITIONS = 4; // warp schedulers per SM

struct warp_schedule {
    int ctas = 0;           // CTAs to launch (at most one per SM)
    int warps_per_cta = 0;
    std::vector<int> first; // per warp (ctas * warps_per_cta + 1 entries): start of its list in `group`
    std::vector<int> group; // group indices, warp after warp
    // warps of a CTA up to the last that has groups in any: the others are not launched and leave their
    // registers to what runs beside
    int warps_used() const
    {
        int used = 0;
        for (size_t w = 0; w + 1 < first.size(); ++w)
            if (first[w + 1] > first[w]) used = std::max(used, static_cast<int>(w) % warps_per_cta + 1);
        return used;
    }
};

// work[g]: cost of group g (points x time steps).  sms: SMs of the device; warps_per_cta: a
// multiple of SUBPARTITIONS.
inline warp_schedule schedule_groups(const std::vector<double> &work, int sms, int warps_per_cta)
{
    warp_schedule ws;
    ws.warps_per_cta = warps_per_cta;
    const int ng = static_cast<int>(work.size());
    if (ng == 0 || sms <= 0 || warps_per_cta < SUBPARTITIONS || warps_per_cta % SUBPARTITIONS) {
        ws.first.assign(1, 0);
        return ws;
    }
    std::vector<int> order(ng);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[a] > work[b]; });

    // bins: sub-partition s of SM c is bin s * sms + c
    const int nbins = sms * SUBPARTITIONS;
    using item = std::pair<double, int>; // (load, index)
    std::priority_queue<item, std::vector<item>, std::greater<item>> heap;
    for (int b = 0; b < nbins; ++b) heap.push({0.0, b});
    std::vector<std::vector<int>> bin_groups(nbins);
    for (int g : order) {
        item top = heap.top();
        heap.pop();
        bin_groups[top.second].push_back(g);
        top.first += work[g];
        heap.push(top);
    }

    // warps of each bin: warp slot * SUBPARTITIONS + s of CTA c
    const int slots = warps_per_cta / SUBPARTITIONS;
    int ctas = 0;
    std::vector<std::vector<int>> warp_groups(static_cast<size_t>(sms) * warps_per_cta);
    for (int b = 0; b < nbins; ++b) {
        if (bin_groups[b].empty()) continue;
        const int s = b / sms, c = b % sms;
        ctas = std::max(ctas, c + 1);
        std::priority_queue<item, std::vector<item>, std::greater<item>> wh;
        for (int j = 0; j < slots; ++j) wh.push({0.0, j});
        for (int g : bin_groups[b]) { // already costliest first
            item top = wh.top();
            wh.pop();
            warp_groups[static_cast<size_t>(c) * warps_per_cta + top.second * SUBPARTITIONS + s].push_back(g);
            top.first += work[g];
            wh.push(top);
        }
    }
    ws.ctas = ctas;
    const size_t nw = static_cast<size_t>(ctas) * warps_per_cta;
    ws.first.assign(nw + 1, 0);
    ws.group.reserve(ng);
    for (size_t w = 0; w < nw; ++w) {
        ws.first[w] = static_cast<int>(ws.group.size());
        ws.group.insert(ws.group.end(), warp_groups[w].begin(), warp_groups[w].end());
    }
    ws.first[nw] = static_cast<int>(ws.group.size());
    return ws;
}

// Lanes per instance (at least `least`) and rows per lane (4 to `most`) of the sweeps in registers, for lines
// whose lanes share `rows` rows: the fewest lanes whose rows fit -- fewer scan levels, or rounds of the
// relay, per row.  (FP64 books that leave the GPU idle ask for as many lanes as their points need: 1000
// calls of 130 points with 128 rows 0.31 ms on 16 lanes, 0.42 on eight, but 60000 11.4 and 8.7.)
inline void register_shape(int rows, int least, int most, int &W, int &R)
{
    W = least;
    while (W * most < rows) W *= 2;
    R = std::max(4, (rows + W - 1) / W);
}

// One group of up to 32 FP64 instances, for memory_limit.
struct group_cost {
    int n, rows, lanes, steps; // points, rows solved, instances, longest time loop
};

// FP64 lines of up to the returned number of points (at most 100: longer ones wait for HBM, and the two
// differ by less than 10 % where the book fills the GPU) take the sweep through memory, longer ones (of up
// to 512 points) the sweep in registers.  The sweep through memory gives a group one warp, which keeps its
// sub-partition's FP64 pipe busy alone; the sweep in registers does more operations per row and spreads a
// group over many warps, two at a time on a sub-partition.  So the latter is the faster as long as the book
// leaves sub-partitions idle (5000 calls of 50 points, 99 steps: 0.36 against 1.06 ms), the former for many
// short lines (60000 calls: 3.1 against 3.4 ms; of 8 points 0.71 against 1.33 ms).  Times of both in us
// per step, fitted to equal calls of 8 to 512 points, 32 to 60000 of them: a group through memory 0.7 +
// 0.196 n (0.218 n of more than 90 points, from HBM); a warp in registers 0.40 + 0.24 R alone, 0.225 + 0.19 R
// of two, the last round of warps taking as long as a whole one.
inline int memory_limit(const std::vector<group_cost> &groups, int sms, int most_rows)
{
    if (sms <= 0) return 0;
    const double parts = 4.0 * sms;
    std::vector<int> order(groups.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return groups[a].n < groups[b].n; });
    struct sum {
        double work = 0.0, longest = 0.0, last = 0.0, warps = 0.0;
    };
    // in registers, the groups from the first of each size on
    std::vector<sum> reg(groups.size() + 1);
    for (size_t q = groups.size(); q-- > 0;) {
        const group_cost &g = groups[order[q]];
        int W = 0, R = 0;
        register_shape(g.rows, 4, most_rows, W, R);
        sum s = reg[q + 1];
        const double units = (g.lanes * W + 31) / 32, wave = 2.0 * (0.225 + 0.19 * R) * g.steps;
        s.work += 0.5 * wave * units / parts;
        s.longest = std::max(s.longest, (0.40 + 0.24 * R) * g.steps);
        s.last = s.warps > 0.0 ? std::min(s.last, wave) : wave;
        s.warps += units;
        reg[q] = s;
    }
    auto reg_time = [&](const sum &s) {
        const double rounds = s.warps / (2.0 * parts);
        return std::max(s.longest, s.work + (rounds > 1.0 ? (std::ceil(rounds) - rounds) * s.last : 0.0));
    };
    double best = reg_time(reg[0]), work = 0.0, longest = 0.0;
    int limit = 0;
    for (size_t q = 0; q < groups.size(); ++q) {
        const group_cost &g = groups[order[q]];
        if (g.n > 100) break;
        const double t = (0.7 + (g.n > 90 ? 0.218 : 0.196) * g.n) * g.steps;
        work += t / parts;
        longest = std::max(longest, t);
        if (q + 1 < groups.size() && groups[order[q + 1]].n == g.n) continue;
        const double mem = work > longest ? work : longest + 0.15 * (q + 1 > parts ? longest : 0.0);
        const double total = mem + reg_time(reg[q + 1]);
        if (total < best) {
            best = total;
            limit = g.n;
        }
    }
    return limit;
}

} // namespace heat1d
} // namespace lss_gb300
