// How the on-chip Gauss-Seidel sweep divides a mesh among the blocks of a
// cluster, and which divisions are worth trying. Host C++ alone: no CUDA.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <utility>
#include <vector>

namespace xg {
namespace host {

// The patches of all instances in slot order (so colour by colour).
struct PatchSet {
    int V = 0, K = 0, ncol = 0;                // vertices, instances, colours
    int per = 8;                               // vertex entries of a patch
    std::vector<int> vert;                     // [P][per], -1 = none
    std::vector<int> colour;                   // [P]
    std::vector<std::vector<int>> mine;        // per instance its patches, ascending
    std::vector<double> centre;                // [P][3] rest centroids
    int patches() const { return (int)colour.size(); }
};

// a division: blocks of an instance, how they are cut, and the estimated time of a sweep
struct ClusterChoice {
    double us;
    int n, shape;
};

class ClusterPartition {
public:
    explicit ClusterPartition(const PatchSet& patches) : s(patches), block(patches.patches(), 0) {}

    std::vector<int> block;  // [P] k n + b: block b of instance k
    std::vector<int> count;  // [K n][ncol] patches of a block and colour

    // Every instance into n blocks; shape 0-2: slabs across that axis, 3:
    // recursive bisection (n a power of two).
    void assign(int shape, int n) {
        if (shape < 3) slabs(shape, n);
        for (int k = 0; shape == 3 && k < s.K; k++) {
            std::vector<int> list = s.mine[k];
            bisect(list, 0, list.size(), k * n, n);
        }
        count.assign((size_t)s.K * n * s.ncol, 0);
        for (int q = 0; q < s.patches(); q++) count[(size_t)block[q] * s.ncol + s.colour[q]]++;
    }

    // colours with a vertex that another block wrote in the colour before: their
    // phases wait for it (about 0.75 us on GB300; a write two phases back is there)
    int stalls() const {
        std::vector<int> first(s.V, -1), last(s.V, -1);
        std::vector<char> w(s.ncol, 0);
        for (int q = 0; q < s.patches(); q++)
            for (int k = 0; k < s.per && vert(q, k) >= 0; k++) {
                const int v = vert(q, k), l = last[v];
                if (l < 0) first[v] = q;
                else if (block[l] != block[q] && s.colour[l] + 1 == s.colour[q]) w[s.colour[q]] = 1;
                last[v] = q;
            }
        for (int v = 0; v < s.V; v++)
            if (last[v] >= 0 && s.colour[first[v]] == 0 && s.colour[last[v]] == s.ncol - 1 &&
                block[first[v]] != block[last[v]])
                w[0] = 1;
        return (int)std::count(w.begin(), w.end(), 1);
    }

    // Whether some vertex lies in more than two blocks. Between two blocks the
    // versions of a vertex alternate, and a block's copy takes them in order:
    // its own writes follow its reads of the other's. A third block's copy would
    // be written by two others, and nothing orders their stores.
    bool crowded() const {
        std::vector<int> one(s.V, -1), two(s.V, -1);
        for (int q = 0; q < s.patches(); q++)
            for (int k = 0; k < s.per && vert(q, k) >= 0; k++) {
                const int v = vert(q, k), b = block[q];
                if (one[v] < 0) one[v] = b;
                else if (one[v] == b || two[v] == b) continue;
                else if (two[v] < 0) two[v] = b;
                else return true;
            }
        return false;
    }

    // The divisions that pay and hold a vertex in two blocks at most, best first.
    // Per round of at most `lanes` patches a block and colour a sweep takes `one`
    // us with one block, `more` with several (and 0.75 where it waits for another
    // block); `other` us a colour is what the route it stands in for takes. most:
    // blocks of a cluster at most; sms: multiprocessors; single: one block only.
    std::vector<ClusterChoice> choices(int lanes, int most, int sms, bool single, double one, double more,
                                       double other) {
        size_t largest = 0;
        for (int k = 0; k < s.K; k++) largest = std::max(largest, s.mine[k].size());
        const size_t unit = (size_t)lanes * s.ncol;
        const int n_min = (int)std::min<size_t>(most, (largest + unit - 1) / unit);
        std::vector<ClusterChoice> out;
        int before = 0;
        for (int n : {n_min, n_min + 1, n_min + 2, n_min + 4, most}) {
            if (n > most || (n > 1 && single) || (s.K > 1 && s.K * n > sms) || n == before) continue;
            before = n;
            for (int shape = 0; shape < 4; shape++) {
                if ((n == 1 && shape > 0) || (shape == 3 && (n & (n - 1)))) continue;
                assign(shape, n);
                double us = 0;
                for (int col = 0; col < s.ncol; col++) {
                    int worst = 1;
                    for (int b = 0; b < s.K * n; b++) worst = std::max(worst, count[(size_t)b * s.ncol + col]);
                    us += (n == 1 ? one : more) * ((worst + lanes - 1) / lanes);
                }
                if (us >= other * s.ncol || (n > 2 && crowded())) continue;
                if (n > 1) us += 0.75 * stalls();
                if (us < other * s.ncol) out.push_back(ClusterChoice{us, n, shape});
            }
        }
        std::stable_sort(out.begin(), out.end(),
                         [](const ClusterChoice& a, const ClusterChoice& b) { return a.us < b.us; });
        return out;
    }

private:
    const PatchSet& s;
    std::vector<std::vector<int>> by_axis[3];

    int vert(int q, int k) const { return s.vert[(size_t)q * s.per + k]; }
    double at(int q, int axis) const { return s.centre[3 * (size_t)q + axis]; }

    // pieces of [first, last) of an instance's patches into blocks b .. b + n - 1
    void bisect(std::vector<int>& list, size_t first, size_t last, int b, int n) {
        if (n == 1) {
            for (size_t i = first; i < last; i++) block[list[i]] = b;
            return;
        }
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (size_t i = first; i < last; i++)
            for (int k = 0; k < 3; k++) {
                lo[k] = std::min(lo[k], at(list[i], k));
                hi[k] = std::max(hi[k], at(list[i], k));
            }
        int ax = 0;
        for (int k = 1; k < 3; k++)
            if (hi[k] - lo[k] > hi[ax] - lo[ax]) ax = k;
        const size_t mid = first + (last - first) / 2;
        std::nth_element(list.begin() + first, list.begin() + mid, list.begin() + last, [&](int a, int d) {
            const double u = at(a, ax), v = at(d, ax);
            return u < v || (u == v && a < d);
        });
        bisect(list, first, mid, b, n / 2);
        bisect(list, mid, last, b + n / 2, n / 2);
    }

    // n slabs across axis ax, the cuts moved to the nearest step of the
    // coordinate (a layer of a grid) within half a slab. An instance of fewer
    // patches than slabs leaves some empty.
    void slabs(int ax, int n) {
        if (by_axis[ax].empty()) {
            by_axis[ax] = s.mine;
            for (auto& l : by_axis[ax])
                std::sort(l.begin(), l.end(),
                          [&](int a, int d) { return at(a, ax) < at(d, ax) || (at(a, ax) == at(d, ax) && a < d); });
        }
        for (int k = 0; k < s.K; k++) {
            const std::vector<int>& l = by_axis[ax][k];
            const long long m = (long long)l.size();
            const double eps = 1e-6 * (at(l.back(), ax) - at(l.front(), ax));
            long long lo = 0;
            for (int r = 0; r < n; r++) {
                long long hi = m * (r + 1) / n;
                for (long long d = 0; r + 1 < n && 2 * n * d <= m; d++) {
                    const long long up = hi + d, down = hi - d;
                    if (up > lo && up < m && at(l[up], ax) - at(l[up - 1], ax) > eps) { hi = up; break; }
                    if (down > lo && at(l[down], ax) - at(l[down - 1], ax) > eps) { hi = down; break; }
                }
                for (long long i = lo; i < hi; i++) block[l[i]] = k * n + r;
                lo = std::max(lo, hi);
            }
        }
    }
};

// Which consecutive instances share the tasks of the dataflow sweeps. A colour of
// a group goes into ceil(m / lanes) tasks, m the patches of its largest colour;
// `warps` warps take the tasks in rounds. count: per instance the patches of each
// colour. Returns the groups' first instances and, last, the number of
// instances: every instance by itself while that costs no round more than fuller
// tasks would, else the smallest groups with the fewest rounds.
inline std::vector<int> task_groups(const std::vector<std::vector<int>>& count, int lanes, long long warps) {
    const int K = (int)count.size();
    auto groups = [&](long long cap, long long& tasks) {  // of at most cap patches of one colour, or one instance
        std::vector<int> first;
        std::vector<long long> sum, with;
        long long m = 0;
        tasks = 0;
        auto close = [&] {
            if (!first.empty()) tasks += std::max(1LL, (m + lanes - 1) / lanes);
        };
        for (int k = 0; k < K; k++) {
            with = sum;
            long long w = 0;
            for (size_t c = 0; c < count[k].size() && !first.empty(); c++) w = std::max(w, with[c] += count[k][c]);
            if (first.empty() || w > cap) {
                close();
                first.push_back(k);
                with.assign(count[k].begin(), count[k].end());
                w = with.empty() ? 0 : *std::max_element(with.begin(), with.end());
            }
            sum.swap(with);
            m = w;
        }
        close();
        first.push_back(K);
        return first;
    };
    long long all = 0, tasks = 0;
    for (const auto& c : count)
        for (int n : c) all += n;
    std::vector<int> best = groups(0, tasks);
    long long rounds = (tasks + warps - 1) / warps;
    for (long long cap = lanes; rounds > 1; cap *= 2) {
        const std::vector<int> g = groups(cap, tasks);
        if ((tasks + warps - 1) / warps < rounds) {
            rounds = (tasks + warps - 1) / warps;
            best = g;
        }
        if (cap > all) break;
    }
    return best;
}

// Whether runs of `lanes` patches keep the colours of a group in step: the k-th
// runs of two colours lie at the same distance in the mesh for every k, to an
// eighth of a run's extent. share: per colour its first patch and how many; pos:
// a patch's place in the mesh order; total: the places of the group.
template <typename Pos>
bool runs_keep_step(const std::vector<std::pair<long long, long long>>& share, int lanes, double total, Pos pos) {
    size_t ref = 0;
    for (size_t c = 1; c < share.size(); c++)
        if (share[c].second > share[ref].second) ref = c;
    double off = 0;  // summed distances from each colour's mean one
    for (const auto& s : share) {
        const long long runs = (s.second + lanes - 1) / lanes;
        auto distance = [&](long long k) {
            return (double)(pos(s.first + lanes * k) - pos(share[ref].first + lanes * k));
        };
        double mean = 0;
        for (long long k = 0; k < runs; k++) mean += distance(k) / (double)runs;
        for (long long k = 0; k < runs; k++) off += std::abs(distance(k) - mean);
    }
    return off * 8 <= total * (double)share.size();  // off / (most colours) against total / most / 8
}

}  // namespace host
}  // namespace xg
