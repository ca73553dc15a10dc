"""How the plane-marching kernels cut axis 0 (gb_split.cuh, compiled here for
the host): chunks lie in the grid for every size, and the rule chooses what
was measured fastest where waves x planes or halving did not."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), os.pardir, 'gpaw_b200', 'csrc')

PROGRAM = r'''
#include <cstdio>
#include "gb_split.cuh"

int main() {
    const long long tiles[] = {1, 2, 7, 64, 147, 148, 149, 592, 593, 5000, 1000000};
    for (int n = 1; n <= 300; n++)
        for (long long t : tiles)
            for (int per_sm = 1; per_sm <= 8; per_sm++)
                for (int step = 1; step <= 2; step++) {
                    const int c = gb::balance_planes(n, step, 6, t, per_sm, 0.2, 1.0);
                    if (c < 1 || c > n) return printf("n %d tiles %lld: chunk %d\n", n, t, c), 1;
                    const int h = gb::halve_planes(n, 4, t, 296);
                    if (h < 1 || h > n) return printf("n %d tiles %lld: half %d\n", n, t, h), 1;
                }
    // 4 x 47 x 63 x 55, restriction of order 6: 3 planes 16.8 us, 2 planes 19.6
    if (gb::balance_planes(23, 2, 11, 16, 3, 0.25, 0.5) != 3) return printf("restriction\n"), 1;
    // 8 x 144^3 complex apply, nn = 1: 36 planes 162 us, 144 planes 218
    if (gb::balance_planes(144, 1, 2, 720, 4, 0.2, 1.0) != 36) return printf("apply\n"), 1;
    // 63^3 residual, nn = 3: 2 planes 8 us, 4 planes 8.6
    if (gb::balance_planes(63, 1, 6, 16, 4, 0.12, 1.0) > 3) return printf("residual\n"), 1;
    return 0;
}
'''


@pytest.mark.skipif(shutil.which('g++') is None, reason='no host compiler')
def test_chunks(tmp_path):
    src, exe = tmp_path / 'chunks.cpp', tmp_path / 'chunks'
    src.write_text(PROGRAM)
    subprocess.run(['g++', '-O2', '-std=c++17', '-I', CSRC, str(src), '-o',
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
