"""The division of the diffusion's difference passes into single vertices and interior vectors:
the index arithmetic of the kernels, run on the host over every cube size from the smallest
allowed one on, with few and many members (vectors are taken from a number of vertices on)."""
import os
import subprocess

from ch_swe_b200.build import ARCH, CSRC, nvcc
from tests.conftest import ROOT

PROGRAM = r"""
#include "chswe.h"
#include "swe_diff.cuh"
#include <cstdio>
#include <vector>
using namespace chswe;
static int split_seen = 0, single_seen = 0;
template <class T, int ORD>
static int check(int N, int members)
{
    constexpr int VW = OV<T>::W;
    const DifSplit s = dif_split<T, ORD>(N, members);
    const int n = N + 1, lo = dif_lo(ORD), P = (N + 1 + 2 * MG + 7) / 8 * 8;
    std::vector<int> seen((size_t)n * n, 0);
    int i, j;
    for (int b = 0; b < s.ne; b++)
        for (int t = 0; t < DIF_NT; t++)
            if (s.nr ? dif_vertex<VW, true>(s, b, t, i, j) : dif_vertex<VW, false>(s, b, t, i, j)) {
                if (i < 1 || i > n || j < 1 || j > n) return 1;
                seen[(size_t)(j - 1) * n + i - 1]++;
            }
    for (int b = 0; b < s.ni; b++)
        for (int t = 0; t < DIF_NT; t++)
            if (dif_vector<VW>(s, b, t, i, j)) {
                // interior rows of both differences at every point; aligned; the neighbour vectors lie in the box
                if (i < lo || i + VW - 1 > n + 1 - lo || j < lo || j > n + 1 - lo || box_off(P, i, j) % VW) return 2;
                if (i - VW + MG - 1 < 0 || i + 2 * VW - 1 + MG - 1 >= P) return 3;
                for (int e = 0; e < VW; e++) seen[(size_t)(j - 1) * n + i - 1 + e]++;
            }
    for (int k : seen)
        if (k != 1) return 4;
    (s.ni ? split_seen : single_seen)++;
    return 0;
}
int main()
{
    for (int members : {1, 4, 64})
        for (int N = 8; N <= 140; N++) {
            int e = check<float, 21>(N, members) + 10 * check<double, 21>(N, members);
            if (N >= 11) e += 100 * check<float, 42>(N, members) + 1000 * check<double, 42>(N, members);
            if (N >= 17) e += 10000 * check<float, 63>(N, members) + 100000 * check<double, 63>(N, members);
            if (e) { printf("N %d members %d: %d\n", N, members, e); return 1; }
        }
    printf("%d %d\n", split_seen, single_seen);
    return 0;
}
"""


def test_every_vertex_is_computed_once(tmp_path):
    src, exe = tmp_path / "split.cu", tmp_path / "split"
    src.write_text(PROGRAM)
    subprocess.run([nvcc(), "-O1", "-std=c++17", *ARCH, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-o", str(exe), str(src)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    split, single = map(int, out.stdout.split())
    assert split > 500 and single > 100
