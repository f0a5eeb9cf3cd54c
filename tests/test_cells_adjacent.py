"""The adjoint's packed comparison of two cells (pbf_adjoint.h) against the
comparison axis by axis: every pair of coordinates along each axis up to the largest
grid, with the other two axes near, at and beyond one cell apart."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mtlphys_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "pbf_adjoint.h"
using namespace mpb;
static long bad = 0, seen = 0, near = 0;
static void check(const int* a, const int* b, bool wide) {
    const bool want = std::abs(a[0] - b[0]) <= 1 && std::abs(a[1] - b[1]) <= 1 && std::abs(a[2] - b[2]) <= 1;
    bad += cells_adjacent(pack_cell(a[0], a[1], a[2]), pack_cell(b[0], b[1], b[2]), wide) != want;
    ++seen;
    near += want;
}
static void grid(int dx, int dy, int dz) {
    const bool wide = wide_grid(dx, dy, dz);
    const int dims[3] = {dx, dy, dz};
    for (int axis = 0; axis < 3; ++axis) {
        const int p = (axis + 1) % 3, q = (axis + 2) % 3;
        const int apart[] = {-3, -2, -1, 0, 1, 2, 3};
        for (int i = 0; i < dims[axis]; ++i)
            for (int j = 0; j < dims[axis]; ++j)
                for (int e = 0; e < 4; ++e) {  // the other axes: a few differences, and the ends of the grid
                    int a[3], b[3];
                    a[axis] = i, b[axis] = j;
                    a[p] = (i * 7 + j) % dims[p], a[q] = (i + 5 * j) % dims[q];
                    b[p] = a[p] + apart[(i + j + e) % 7], b[q] = a[q] + apart[(i * 3 + j + 2 * e) % 7];
                    if (e == 2) a[p] = 0, b[p] = dims[p] - 1;
                    if (e == 3) a[p] = dims[p] - 1, b[p] = 0, a[q] = 0, b[q] = dims[q] - 1;
                    if (b[p] < 0 || b[p] >= dims[p] || b[q] < 0 || b[q] >= dims[q]) continue;
                    check(a, b, wide);
                }
    }
}
int main() {
    grid(2045, 2045, 1021);  // the largest that is not wide
    grid(2046, 2045, 1021);
    grid(2048, 2048, 1024);  // the largest
    grid(86, 86, 86);
    std::printf("%ld %ld %ld %d%d%d\n", bad, seen, near, wide_grid(2045, 2045, 1021), wide_grid(2045, 2046, 3),
                wide_grid(2, 2, 1022));
}
"""


def test_packed_comparison_equals_the_one_axis_by_axis(tmp_path):
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", "t.cpp", "-o", "t"],
                   cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    bad, seen, near = map(int, out[:3])
    assert bad == 0 and seen > 10_000_000 and near > 1000
    assert out[3] == "011"
