"""What the linear pass stages (gb_stage.cuh, compiled here for the host):
for short and long sides, every boundary and half-width, no cell lies outside
the plane, and each cell that a point of the plane reads holds the value its
boundary gives."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), os.pardir, 'gpaw_b200', 'csrc')

# every tile of an n1 x n2 plane, tx columns wide (32 double, 64 float):
# prints the first cell that is wrong
PROGRAM = r'''
#include <cstdio>
#include "gb_stage.cuh"

static int bad(const char* what, int n1, int n2, int per, int nn, int tx, int r, int c, int at) {
    printf("%s: plane %d x %d periodic %d nn %d tile %d: cell (%d, %d) -> %d\n", what, n1, n2,
           per, nn, tx, r, c, at);
    return 1;
}

static int wrap(int j, int n, int per) { return per ? (j % n + n) % n : j < 0 || j >= n ? -1 : j; }

static int plane(int n1, int n2, int per, int nn, int tx) {
    const int p1 = per & 1, p2 = per >> 1;
    for (int y0 = 0; y0 < n1; y0 += gb::PT_ROWS)
        for (int x0 = 0; x0 < n2; x0 += tx)
            for (int r = y0 - nn; r < y0 + gb::PT_ROWS + nn; r++)
                for (int c = x0 - gb::PT_HX; c < x0 + tx + gb::PT_HX; c++) {
                    const int at = gb::staged_offset(r, c, n1, n2, p1, p2);
                    if (at < -1 || at >= n1 * n2)
                        return bad("outside the plane", n1, n2, per, nn, tx, r, c, at);
                    // read by a point of the plane along one axis
                    const bool row = r >= 0 && r < n1 && c >= -nn && c < n2 + nn;
                    const bool col = c >= 0 && c < n2 && r >= -nn && r < n1 + nn;
                    if (!row && !col) continue;
                    const int wr = wrap(r, n1, p1), wc = wrap(c, n2, p2);
                    if (at != (wr < 0 || wc < 0 ? -1 : wr * n2 + wc))
                        return bad("wrong value", n1, n2, per, nn, tx, r, c, at);
                }
    return 0;
}

int main() {
    for (int nn = 1; nn <= 3; nn++)
        for (int tx = 32; tx <= 64; tx *= 2)
            for (int per = 0; per < 4; per++)
                for (int n1 = nn; n1 <= 40; n1++)
                    for (int n2 = gb::PT_HX; n2 <= 70; n2++)
                        if (plane(n1, n2, per, nn, tx)) return 1;
    return 0;
}
'''


@pytest.mark.skipif(shutil.which('g++') is None, reason='no host compiler')
def test_staged_cells_lie_in_the_plane(tmp_path):
    src, exe = tmp_path / 'stage.cpp', tmp_path / 'stage'
    src.write_text(PROGRAM)
    subprocess.run(['g++', '-O2', '-std=c++17', '-x', 'c++', '-I', CSRC,
                    str(src), '-o', str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
