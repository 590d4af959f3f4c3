"""How the on-chip sweep divides a mesh among the blocks of a cluster
(csrc/xpbd_partition.hpp, host C++ alone), compiled here with the standard
library's index checks on."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
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

int main(int argc, char** argv) {
    const int K = std::atoi(argv[1]), nx = std::atoi(argv[2]), ny = std::atoi(argv[3]), nz = std::atoi(argv[4]);
    const PatchSet s = grid(K, nx, ny, nz);
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
    for (const ClusterChoice& c : p.choices(128, 16, 152, false, 1.1, 1.4, 2.2))
        std::printf("%d %d %.2f\n", c.n, c.shape, c.us);
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
