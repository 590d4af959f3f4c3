"""How the on-chip sweep divides a mesh among the blocks of a cluster
(csrc/xpbd_partition.hpp, host C++ alone), compiled here with the standard
library's index checks on."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include "xpbd_partition.hpp"
using namespace xg::host;

// a grid of hex patches, one a hex, coloured by parity (slot order: colour by colour)
static PatchSet grid(int K, int nx, int ny, int nz) {
    PatchSet s;
    s.K = K; s.ncol = (nx > 1 ? 2 : 1) * (ny > 1 ? 2 : 1) * (nz > 1 ? 2 : 1);
    s.mine.resize(K);
    const int VI = (nx + 1) * (ny + 1) * (nz + 1);
    s.V = K * VI;
    for (int c = 0; c < s.ncol; c++)
        for (int k = 0; k < K; k++)
            for (int j = 0; j < ny; j++)
                for (int i = 0; i < nx; i++)
                    for (int l = 0; l < nz; l++) {
                        int col = 0, bit = 1;
                        if (nz > 1) { col += bit * (l & 1); bit *= 2; }
                        if (nx > 1) { col += bit * (i & 1); bit *= 2; }
                        if (ny > 1) col += bit * (j & 1);
                        if (col != c) continue;
                        s.mine[k].push_back((int)s.colour.size());
                        s.colour.push_back(c);
                        for (int d = 0; d < 8; d++)
                            s.vert.push_back(k * VI + (l + (d & 1)) + (i + (d >> 1 & 1)) * (nz + 1) +
                                             (j + (d >> 2)) * (nz + 1) * (nx + 1));
                        s.centre.push_back(i + 0.5); s.centre.push_back(j + 0.5); s.centre.push_back(l + 0.5);
                    }
    return s;
}

// n patches of up to eight of the vertices around a random point, coloured greedily
static PatchSet cloud(int n) {
    PatchSet s;
    s.K = 1; s.V = 2 * n;
    std::mt19937 rng(5);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    std::vector<double> X(3 * s.V);
    for (double& x : X) x = u(rng);
    std::vector<std::vector<int>> items(n);
    std::vector<double> at(3 * n);
    std::vector<int> col(n), order(s.V);
    std::vector<std::vector<char>> used(s.V, std::vector<char>(256, 0));
    for (int q = 0; q < n; q++) {
        for (int k = 0; k < 3; k++) at[3 * q + k] = u(rng);
        for (int v = 0; v < s.V; v++) order[v] = v;
        auto dist = [&](int v) {
            double d = 0;
            for (int k = 0; k < 3; k++) d += (X[3 * v + k] - at[3 * q + k]) * (X[3 * v + k] - at[3 * q + k]);
            return d;
        };
        const int m = 4 + q % 5;
        std::partial_sort(order.begin(), order.begin() + m, order.end(), [&](int a, int b) { return dist(a) < dist(b); });
        items[q].assign(order.begin(), order.begin() + m);
        int c = 0;
        for (bool again = true; again;) {
            again = false;
            for (int v : items[q]) again = again || used[v][c];
            if (again) c++;
        }
        for (int v : items[q]) used[v][c] = 1;
        col[q] = c;
        s.ncol = std::max(s.ncol, c + 1);
    }
    s.mine.resize(1);
    for (int c = 0; c < s.ncol; c++)
        for (int q = 0; q < n; q++) {
            if (col[q] != c) continue;
            s.mine[0].push_back((int)s.colour.size());
            s.colour.push_back(c);
            for (int k = 0; k < 8; k++) s.vert.push_back(k < (int)items[q].size() ? items[q][k] : -1);
            for (int k = 0; k < 3; k++) s.centre.push_back(at[3 * q + k]);
        }
    return s;
}

int main(int argc, char** argv) {
    const int K = std::atoi(argv[1]), nx = std::atoi(argv[2]), ny = std::atoi(argv[3]), nz = std::atoi(argv[4]);
    const PatchSet s = K ? grid(std::abs(K), nx, ny, nz) : cloud(nx);
    if (K < 0) {  // whether runs of 32 patches keep the colours in step
        std::vector<std::pair<long long, long long>> share(s.ncol, {0, 0});
        std::vector<int> pos(s.patches());
        for (int q = 0; q < s.patches(); q++) {
            if (share[s.colour[q]].second++ == 0) share[s.colour[q]].first = q;
            const double* c = &s.centre[3 * (size_t)q];
            pos[q] = 5 * ((int)c[2] + nz * ((int)c[0] + nx * (int)c[1]));
        }
        std::printf("%d", (int)runs_keep_step(share, 32, 5.0 * nx * ny * nz, [&](long long q) { return pos[q]; }));
        return 0;
    }
    ClusterPartition p(s);
    for (int n = 1; n <= 16; n++)
        for (int shape = 0; shape < 4; shape++) {
            if (shape == 3 && (n & (n - 1))) continue;
            p.assign(shape, n);
            for (int k = 0; k < K; k++)
                for (int q : s.mine[k])
                    if (p.block[q] < k * n || p.block[q] >= (k + 1) * n) return 1;
            p.stalls();
        }
    for (const ClusterChoice& c : p.choices(128, 16, 152, false, 1.1, 1.4, 2.2)) {
        p.assign(c.shape, c.n);
        size_t most = 0;  // blocks that hold one vertex
        std::vector<std::vector<int>> in(s.V);
        for (int q = 0; q < s.patches(); q++)
            for (int k = 0; k < 8 && s.vert[8 * (size_t)q + k] >= 0; k++) {
                std::vector<int>& l = in[s.vert[8 * (size_t)q + k]];
                if (std::find(l.begin(), l.end(), p.block[q]) == l.end()) l.push_back(p.block[q]);
                most = std::max(most, l.size());
            }
        std::printf("%d %d %.2f %zu\n", c.n, c.shape, c.us, most);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("partition")
    src, exe = str(d / "p.cpp"), str(d / "p")
    open(src, "w").write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GLIBCXX_ASSERTIONS", "-I",
                    os.path.join(ROOT, "xpbd-tissue-sim_gb300", "csrc"), src, "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("K,dims", [(1, (1, 1, 1)), (1, (2, 1, 1)), (1, (2, 2, 2)), (1, (3, 5, 1)), (3, (1, 2, 1)),
                                    (1, (17, 3, 2))])
def test_partition_of_fewer_patches_than_blocks(planner, K, dims):
    """Every candidate division of a mesh with fewer patches than a cluster has
    blocks reads inside its lists and keeps each instance in its own blocks."""
    r = subprocess.run([planner, str(K), *map(str, dims)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("K,dims", [(1, (24, 24, 24)), (1, (20, 35, 20)), (1, (19, 33, 19)), (1, (10, 100, 10)),
                                    (1, (20, 20, 20)), (1, (1, 40, 1)), (7, (10, 10, 10)), (5, (14, 14, 14)),
                                    (0, (1500, 0, 0)), (0, (4000, 0, 0))])
def test_no_vertex_lies_in_more_than_two_blocks(planner, K, dims):
    """A vertex's copies are written without a fence between the blocks, which
    keeps its versions in order for two holders and not for three. K = 0: an
    unstructured set of patches."""
    r = subprocess.run([planner, str(K), *map(str, dims)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert all(int(most) <= 2 for _, _, _, most in rows), rows
    if K == 1 and dims == (10, 100, 10):  # the beam keeps its slabs
        assert rows[0][:2] == ["10", "1"]


GROUPS = r"""
#include <cstdio>
#include <cstdlib>
#include "xpbd_partition.hpp"
// stdin: warps, K, ncol, counts by instance; out: the groups' first instances and K
int main() {
    long long warps;
    int K, ncol;
    if (std::scanf("%lld %d %d", &warps, &K, &ncol) != 3) return 2;
    std::vector<std::vector<int>> n(K, std::vector<int>(ncol));
    for (auto& r : n)
        for (int& v : r)
            if (std::scanf("%d", &v) != 1) return 2;
    for (int g : xg::host::task_groups(n, 32, warps)) std::printf("%d ", g);
    return 0;
}
"""


@pytest.fixture(scope="module")
def grouper(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    src, exe = str(d / "g.cpp"), str(d / "g")
    open(src, "w").write(GROUPS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GLIBCXX_ASSERTIONS", "-I",
                    os.path.join(ROOT, "xpbd-tissue-sim_gb300", "csrc"), src, "-o", exe], check=True)
    return exe


def _rounds(counts, first, warps):
    tasks = sum(max(1, -(-int(counts[a:b].sum(0).max()) // 32)) for a, b in zip(first[:-1], first[1:]))
    return -(-tasks // warps)


@pytest.mark.parametrize("name,warps", [("tiny", 1216), ("tiny", 1), ("uneven", 1216), ("just_over", 1216),
                                        ("mixed", 1216), ("one", 1216), ("odd_colours", 100)])
def test_small_instances_share_tasks_only_where_that_saves_rounds(grouper, name, warps):
    """Tasks of the dataflow sweeps: never more rounds of the warps than equal
    shares of the union of all instances take; every instance by itself where
    that costs no round more."""
    rng = np.random.default_rng(0)
    counts = {"tiny": np.tile([6, 4, 4, 4, 6, 4, 4, 2], (5000, 1)),       # 40 hexes each
              "uneven": rng.integers(40, 1800, (96, 1)) + rng.integers(0, 9, (96, 8)),
              "just_over": np.tile([40, 36, 36, 32, 40, 36, 36, 32], (700, 1)),
              "mixed": np.concatenate([np.full((2000, 8), 3), np.full((3, 8), 9000)]),
              "one": np.full((1, 8), 32768),
              "odd_colours": rng.integers(0, 50, (640, 13))}[name]
    text = f"{warps} {len(counts)} {counts.shape[1]} " + " ".join(map(str, counts.ravel()))
    r = subprocess.run([grouper], input=text, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    first = [int(v) for v in r.stdout.split()]
    assert first[0] == 0 and first[-1] == len(counts) and all(b > a for a, b in zip(first, first[1:]))
    got, union = _rounds(counts, first, warps), _rounds(counts, [0, len(counts)], warps)
    alone = _rounds(counts, list(range(len(counts) + 1)), warps)
    assert got <= min(union, alone)
    if alone == union:
        assert len(first) == len(counts) + 1
    if name in ("tiny", "just_over") and warps > 1:
        assert got < alone


@pytest.mark.parametrize("dims,runs", [((48, 48, 48), 1), ((26, 60, 26), 1), ((36, 35, 36), 1), ((36, 27, 28), 1),
                                       ((2, 2, 2), 1), ((35, 36, 36), 0), ((36, 36, 35), 0), ((16, 16, 15), 0),
                                       ((47, 49, 45), 0), ((29, 29, 28), 0)])
def test_runs_of_32_patches_only_where_they_keep_the_colours_in_step(planner, dims, runs):
    """The mesh order runs along z, then x, then y: an odd number of hexes along y
    ends some colours a layer earlier, along x or z it lets them drift apart."""
    r = subprocess.run([planner, "-1", *map(str, dims)], capture_output=True, text=True)
    assert r.returncode == 0 and int(r.stdout) == runs, r.stderr
