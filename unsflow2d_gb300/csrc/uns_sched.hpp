// uns_sched.hpp -- host-side warp schedule of the LU-SGS sweeps.
//
// The forward sweep of lusgs2 (CCFVM/lusgs.F90:245-280, NCFVM/lusgs.f90:48-86)
// updates entity i from its already-updated neighbours j < i; the backward
// sweep (CCFVM/lusgs.F90:283-318, NCFVM/lusgs.f90:88-124) from j > i and from
// i's own forward value.  Each (entity, pass) is one item of a DAG whose
// longest path is long (thousands of items on an O-mesh), so the sweep is
// latency-bound: what matters is how fast one item can follow another.
//
// An item that follows a predecessor computed by the same warp takes its
// values from registers; one that follows an item of another warp of its block
// reads them in shared memory; one that follows another block's must see the
// published record in L2.  list_schedule assigns the items to warps by greedy
// list scheduling on that cost model (an item costs kCompute, an edge between
// warps of a block kNear, between blocks kSync): each item, in topological
// order, goes to the warp that starts it earliest among those of its
// predecessors whose newest item that is, the warps of its predecessors'
// blocks, and the warp that frees up first.
//
// Costs by measurement and replay (NCFVM 1024x512, hand-offs of 0.1 of an item
// inside a block and 0.55 between blocks, in levels of the graph): 1.27 with
// one cost for every edge and no preference for a block, 1.13 with 0.05 and
// 0.30 as below, 1.17 with the hand-offs' own 0.1 and 0.55, which spread the
// chains less.
//
// Each warp's list is in increasing simulated start time and every
// dependency of an item has a strictly earlier simulated start, so with all
// warps resident (cooperative launch) the lowest-start unfinished item can
// always proceed: the sweep cannot deadlock.
#pragma once
#include <algorithm>
#include <vector>

namespace uns {

constexpr int kSrcBits = 28;  // of WarpSchedule::src: the list index, under the warp of the block

struct WarpSchedule {
    std::vector<int> off;    // nwarps + 1 offsets into items
    std::vector<int> items;  // (entity << 1) | pass, pass 0 = forward, 1 = backward
    // Item by item, for each neighbour that the item waits for (in the order of
    // its CSR list): where its sweep warp finds the neighbour's record, (warp of
    // the block << kSrcBits) | list index, or -1 for one of another block, in L2.
    std::vector<int> src;
    double makespan = 0.0;   // simulated length in units of one item's compute
    int nlev_fwd = 0, nlev_bwd = 0;

    // The blocks that have items: the launch needs no others.
    int blocks() const;
    // Whether every list index fits in src.
    bool indexable() const;
};

constexpr int kSchedGroup = 4;  // consecutive warps of a block
static_assert(kSchedGroup <= 4, "WarpSchedule::src has two bits for the warp");
constexpr int kSideBySide = 3;  // sweeps of separate handles that should fit beside each other

// How many of nwarps warps the lists of 2 n items in `levels` dependency levels
// are spread over.  Two warps per item of an average level keep the chain
// within 3 % of what all the warps give it (NCFVM sweeps, 92 items per level:
// 1.83 ms on 608 warps, 1.87 on 200; 147 items: 2.99 and, on 304, 3.01), so a
// graph narrow enough takes a half or a third of the blocks and leaves the
// other SMs to other handles' sweeps: three solves of the first mesh in three
// threads 5.49 -> 2.18 ms per iteration.
inline int sweep_warps(int n, int levels, int nwarps) {
    const long long side = n > 0 ? std::min<long long>(kSideBySide, (long long)nwarps * levels / (4LL * n)) : 1;
    if (side < 2) return nwarps;
    return std::min(nwarps, std::max(1, nwarps / kSchedGroup / (int)side) * kSchedGroup);
}

// nbr_off / nbr: CSR neighbour lists of the n entities (any order, entries
// outside [0, n) ignored).  nwarps: warps of the cooperative launch.  kNear,
// kSync: the extra delay of a dependency on another warp of the block and of
// another block, in units of one item's compute.  sweep_warps of them get items.
inline WarpSchedule list_schedule(int n, const int* nbr_off, const int* nbr, int nwarps, double kNear = 0.05,
                                  double kSync = 0.30) {
    constexpr double kCompute = 1.0;
    // Topological orders: forward by dependency level (then index), backward
    // by backward level (then descending index).
    std::vector<int> lev(n, 0), levb(n, 0);
    int nlev = 0, nlevb = 0;
    for (int i = 0; i < n; ++i) {
        int l = 0;
        for (int k = nbr_off[i]; k < nbr_off[i + 1]; ++k) {
            int j = nbr[k];
            if (j >= 0 && j < i) l = std::max(l, lev[j] + 1);
        }
        lev[i] = l;
        nlev = std::max(nlev, l + 1);
    }
    for (int i = n - 1; i >= 0; --i) {
        int l = 0;
        for (int k = nbr_off[i]; k < nbr_off[i + 1]; ++k) {
            int j = nbr[k];
            if (j > i && j < n) l = std::max(l, levb[j] + 1);
        }
        levb[i] = l;
        nlevb = std::max(nlevb, l + 1);
    }
    std::vector<int> fwd(n), bwd(n);
    {
        std::vector<int> cnt(nlev + 1, 0);
        for (int i = 0; i < n; ++i) ++cnt[lev[i] + 1];
        for (int l = 0; l < nlev; ++l) cnt[l + 1] += cnt[l];
        for (int i = 0; i < n; ++i) fwd[cnt[lev[i]]++] = i;
        std::vector<int> cb(nlevb + 1, 0);
        for (int i = 0; i < n; ++i) ++cb[levb[i] + 1];
        for (int l = 0; l < nlevb; ++l) cb[l + 1] += cb[l];
        for (int i = n - 1; i >= 0; --i) bwd[cb[levb[i]]++] = i;
    }

    struct Item {  // a placed item: its simulated finish, warp and place in the warp's list
        double fin;
        int warp, index;
    };
    std::vector<Item> done(2 * (size_t)n);
    const int used = sweep_warps(n, nlev + nlevb, nwarps);
    std::vector<double> wfree(nwarps, 0.0);
    std::vector<int> wlast(nwarps, -1);
    std::vector<int> count(nwarps, 0), codes, srcs;  // items per warp; every item and its sources as they are placed
    std::vector<int> nsrc(nwarps, 0);
    codes.reserve(2 * (size_t)n);
    srcs.reserve(nbr_off[n] - nbr_off[0]);
    // The warp that frees up first (of several, the lowest): a tournament.  A
    // heap with an entry per placement outgrows the caches on a large mesh
    // (4.2 M cells).
    int leaves = 1;
    while (leaves < used) leaves *= 2;
    std::vector<int> first(2 * (size_t)leaves, -1);
    auto earlier = [&](int a, int b) { return b < 0 || (a >= 0 && wfree[a] <= wfree[b]) ? a : b; };
    for (int w = 0; w < used; ++w) first[leaves + w] = w;
    for (int k = leaves - 1; k > 0; --k) first[k] = earlier(first[2 * k], first[2 * k + 1]);

    std::vector<int> preds;
    std::vector<Item> pr;  // the predecessors' items
    double makespan = 0.0;
    auto place = [&](int code) {
        pr.clear();
        double last = 0.0;
        for (int p : preds) { pr.push_back(done[p]); last = std::max(last, done[p].fin); }
        // The item's start on warp c, and the candidates: a warp that is not
        // free before the best start so far cannot improve on it.
        int w = -1;
        double s = 0.0;
        auto consider = [&](int c) {
            double t = wfree[c];
            if (w >= 0 && std::max(t, last) >= s - 1e-12) return;
            for (const Item& p : pr)
                t = std::max(t, p.fin + (p.warp == c ? 0.0 : (p.warp / kSchedGroup == c / kSchedGroup ? kNear : kSync)));
            if (w < 0 || t < s - 1e-12) { w = c; s = t; }
        };
        for (size_t k = 0; k < pr.size(); ++k)
            if (wlast[pr[k].warp] == preds[k]) consider(pr[k].warp);
        for (size_t k = 0; k < pr.size(); ++k) {
            const int g = pr[k].warp / kSchedGroup;
            bool again = false;
            for (size_t q = 0; q < k; ++q) again = again || pr[q].warp / kSchedGroup == g;
            if (again) continue;
            for (int c = g * kSchedGroup; c < (g + 1) * kSchedGroup && c < used; ++c) consider(c);
        }
        consider(first[1]);
        done[code] = {s + kCompute, w, count[w]++};
        makespan = std::max(makespan, s + kCompute);
        wfree[w] = s + kCompute;
        wlast[w] = code;
        // w frees up later than before: only the rounds that it had won change
        for (int k = (leaves + w) / 2; k > 0 && first[k] == w; k /= 2) first[k] = earlier(first[2 * k], first[2 * k + 1]);
        codes.push_back(code);
        for (size_t k = code & 1; k < pr.size(); ++k)  // not a backward item's own forward value
            srcs.push_back(pr[k].warp / kSchedGroup == w / kSchedGroup ? (pr[k].warp % kSchedGroup) << kSrcBits | pr[k].index : -1);
        nsrc[w] += (int)pr.size() - (code & 1);
    };
    for (int i : fwd) {
        preds.clear();
        for (int k = nbr_off[i]; k < nbr_off[i + 1]; ++k) {
            int j = nbr[k];
            if (j >= 0 && j < i) preds.push_back(2 * j);
        }
        place(2 * i);
    }
    for (int i : bwd) {
        preds.clear();
        preds.push_back(2 * i);  // own forward value
        for (int k = nbr_off[i]; k < nbr_off[i + 1]; ++k) {
            int j = nbr[k];
            if (j > i && j < n) preds.push_back(2 * j + 1);
        }
        place(2 * i + 1);
    }
    WarpSchedule out;
    out.makespan = makespan;
    out.nlev_fwd = nlev;
    out.nlev_bwd = nlevb;
    out.off.assign(nwarps + 1, 0);
    std::vector<int> at(nwarps + 1, 0);  // where each warp's sources go
    for (int w = 0; w < nwarps; ++w) {
        out.off[w + 1] = out.off[w] + count[w];
        at[w + 1] = at[w] + nsrc[w];
    }
    out.items.resize(codes.size());
    out.src.resize(srcs.size());
    size_t from = 0;
    for (int code : codes) {
        const Item& d = done[code];
        out.items[out.off[d.warp] + d.index] = code;
        const int i = code >> 1, pass = code & 1;
        for (int k = nbr_off[i]; k < nbr_off[i + 1]; ++k) {
            const int j = nbr[k];
            if (j >= 0 && j < n && (pass == 0 ? j < i : j > i)) out.src[at[d.warp]++] = srcs[from++];
        }
    }
    return out;
}

// The bound of a wait inside a sweep block for a wait limit of `wait` cycles on
// another block's record: longer than that wait, so that the warp whose record
// does not come is the one to report it.  (A limit of any size: no overflow.)
constexpr long long ring_wait_limit(long long wait) {
    constexpr long long kMost = 0x7fffffffffffffffLL, kExtra = 100000000LL;
    return wait > (kMost - kExtra) / 4 ? kMost : 4 * wait + kExtra;
}

inline int WarpSchedule::blocks() const {
    int w = (int)off.size() - 1;
    while (w > 0 && off[w] == off[w - 1]) --w;
    return std::max(1, (w + kSchedGroup - 1) / kSchedGroup);
}

inline bool WarpSchedule::indexable() const {
    for (size_t w = 0; w + 1 < off.size(); ++w)
        if (off[w + 1] - off[w] > 1 << kSrcBits) return false;
    return true;
}

// Asks for what the records of some later item are made of: a warp's list jumps
// over the whole mesh (CCFVM, 4.2 M cells: the records 1.1 -> 0.64 s).
inline void ask_ahead(const WarpSchedule& ws, size_t pos, const int* off, const int* nbr, const int* edge, const signed char* side) {
    if (pos + 32 < ws.items.size()) __builtin_prefetch(off + (ws.items[pos + 32] >> 1));
    if (pos + 16 < ws.items.size()) {
        const int k = off[ws.items[pos + 16] >> 1];
        __builtin_prefetch(nbr + k);
        __builtin_prefetch(edge + k);
        __builtin_prefetch(side + k);
    }
}

}  // namespace uns
