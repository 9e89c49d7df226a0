"""What a scratch for every shorter sequence holds beside the planes: bounds on the partial results of a split backward, against the
splits themselves (csrc/tc_split.cuh, compiled here; without a device it takes a B200's 148 SMs)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "z-transformer_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include "tc_split.cuh"
int main() {
    long long splits = 0, over = 0;
    const int heads[][2] = {{1, 1}, {2, 1}, {4, 2}, {6, 2}, {8, 2}, {12, 4}, {16, 16}, {32, 8}, {32, 1}, {64, 2}};
    for (const auto &h : heads)
        for (int batch : {1, 2, 3, 7})
            for (int dim : {32, 64, 80, 128}) {
                size_t most = 0;  // of this length and every shorter one
                for (int T = 1; T <= 2600; T += T < 600 ? 1 : 37) {
                    const size_t floats = zt::bwd_parts_floats(batch, T, h[0], h[1], dim);
                    splits += floats > 0;
                    if (floats > most) most = floats;
                    if (most <= zt::bwd_parts_floats_bound(batch, T, h[0], dim)) continue;
                    if (over++ < 5) printf("batch %d, T %d, %d/%d heads of %d: %zu floats, bound %zu\n", batch, T, h[0], h[1], dim, most,
                                           zt::bwd_parts_floats_bound(batch, T, h[0], dim));
                }
            }
    printf("%lld splits, %lld over\n", splits, over);
    return over > 0 || splits < 10000;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_a_split_backwards_parts_fit_their_bound(tmp_path):
    src = tmp_path / "bounds.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "bounds")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", exe, str(src)])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
