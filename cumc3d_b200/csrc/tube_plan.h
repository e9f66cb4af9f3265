// tube_plan.h -- which problems of a batch run on clusters of their own
// (tube_kernel.cuh) and which in the persistent kernel (batch_kernel.cuh).
// Host code without CUDA, so that it is tested without a device.
#pragma once
#include <vector>

namespace cumc {

// problems first .. first + count - 1 of the launch order (largest first), one
// cluster of `size` CTAs each, of 254 cells (wide) or 126; size 0: the
// persistent kernel
struct TubeLaunch {
    int first, count, size;
    bool wide;
};

// Every problem of up to 16 x 254 cells gets a cluster of its own, one cell per
// thread: the fewest CTAs that hold it, a power of two.  CTAs
// of 254 cells keep the most cells in flight; a batch whose CTAs are all
// resident at once (two an SM) waits for its largest problems, and those run
// sooner on CTAs of 126 cells (PPM FP64, wide and narrow: 64 problems of 128 to
// 2048 cells, 1.6 CTAs an SM, 14.0 and 10.9 ms; 128, 3.3 an SM, 14.8 and 15.4;
// 512 of 128 to 4096, 22 an SM, 163 and 179).  A batch that leaves half the
// SMs idle takes twice as many CTAs (up to 8, at least 16 cells each): a CTA
// with fewer warps runs a stage sooner.  Problems with the same cluster are
// neighbours in the launch order; each such class is one launch.
inline std::vector<TubeLaunch> tube_plan(const std::vector<int> &sorted_n, int sm_count) {
    const int np = (int)sorted_n.size(), most = 16 * 254;
    int big = 0;  // problems beyond 16 CTAs
    while (big < np && sorted_n[big] > most) ++big;
    auto ctas = [&](int n, int cells) {
        int c = 1;
        while (c < 16 && (n + c - 1) / c > cells) c *= 2;
        return c;
    };
    long long total = 0;
    for (int p = big; p < np; ++p) total += ctas(sorted_n[p], 254);
    const bool narrow = total <= 2LL * sm_count;
    auto wide_of = [&](int n) { return !narrow || n > 16 * 126; };
    if (narrow) {
        total = 0;
        for (int p = big; p < np; ++p) total += ctas(sorted_n[p], wide_of(sorted_n[p]) ? 254 : 126);
    }
    int wider = 1;
    while (wider < 8 && 2 * wider * total <= sm_count) wider *= 2;
    auto size_of = [&](int n) {
        int c = ctas(n, wide_of(n) ? 254 : 126);
        for (int w = wider; w > 1 && c < 8 && n / (2 * c) >= 16; w /= 2) c *= 2;
        return c;
    };
    std::vector<TubeLaunch> plan;
    if (big > 0) plan.push_back({0, big, 0, false});
    for (int p = big; p < np;) {
        const int size = size_of(sorted_n[p]);
        const bool wide = wide_of(sorted_n[p]);
        int q = p;
        while (q < np && size_of(sorted_n[q]) == size && wide_of(sorted_n[q]) == wide) ++q;
        plan.push_back({p, q - p, size, wide});
        p = q;
    }
    return plan;
}

// Launches a plan: tube(launch) says whether the device took the class,
// persistent(first, count) whether the persistent kernel did.  A class that is
// refused, of any size (a device may have no room for its clusters), joins the
// problems too large for a cluster; neighbours share a call.
template <class Tube, class Persistent>
inline bool run_plan(const std::vector<TubeLaunch> &plan, Tube tube, Persistent persistent) {
    std::vector<TubeLaunch> rest;
    for (const TubeLaunch &l : plan) {
        if (l.size > 0 && tube(l)) continue;
        if (!rest.empty() && rest.back().first + rest.back().count == l.first) rest.back().count += l.count;
        else rest.push_back(l);
    }
    for (const TubeLaunch &l : rest)
        if (!persistent(l.first, l.count)) return false;
    return true;
}

}  // namespace cumc
