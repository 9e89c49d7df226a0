"""The order of the wide backward's products (csrc/tc_bwd_wide.cuh, compiled here): every unit once in either order, and a head's units
in turn only where that makes no block longer by more than a tenth."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "z-transformer_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <set>
#include "tc_bwd_wide.cuh"
using namespace zt;
// the longest block's steps of MMAs, with two more for a unit's start and end; -1 where a unit is missing or there twice
static long long longest(tcw::WideParams p, bool in_turn, int blocks) {
    p.in_turn = in_turn;
    const int n = 3 * (p.Tp / 128) * p.units * p.pieces;
    std::set<long long> seen;
    long long most = 0;
    for (int first = 0; first < blocks && first < n; ++first) {
        long long steps = 0;
        for (int i = first; i < n; i += blocks) {
            const tcw::TriUnit u(p, i);
            seen.insert((((long long)u.which * p.units + u.u) * p.pieces + u.k_begin / tcw::kPiece) * (p.Tp / 128) + u.m0 / 128);
            if (u.n_steps > 0) steps += u.n_steps + 2;
        }
        if (steps > most) most = steps;
    }
    return p.pieces > 1 || (int)seen.size() == n ? most : -1;
}
int main() {
    const int blocks = 148;
    int bad = 0, turns = 0, others = 0;
    for (int nt = 1; nt <= 8; ++nt)
        for (int units = 1; units <= 320; units += units < 80 ? 1 : 16) {
            tcw::WideParams p{};
            p.T = p.Tp = nt * 128, p.units = units, p.pieces = 1, p.n_heads = 4, p.n_kv_heads = 2;
            const bool turn = tcw::products_in_turn(1, nt, units, blocks);
            const long long in_turn = longest(p, true, blocks), by_product = longest(p, false, blocks);
            (turn ? turns : others)++;
            if (in_turn < 0 || by_product < 0 || (turn && in_turn * 10 > by_product * 11))
                ++bad, printf("T %d, %d heads: in turn %lld, by product %lld\n", p.T, units, in_turn, by_product);
        }
    return bad > 0 || turns < 100 || others < 100 || tcw::products_in_turn(2, 8, 1 << 20, blocks);
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_every_unit_once_and_no_block_far_longer_in_turn(tmp_path):
    src = tmp_path / "order.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "order")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", exe, str(src), "-lcuda"])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
