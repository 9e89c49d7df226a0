"""What the one-launch pre-passes are planned to be (csrc/prepass.cuh, compiled here; without a device it takes a B200's 148 SMs): a cluster has a
unit, or a step, for each of its blocks, whichever tensor they convert."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "z-transformer_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
pytestmark = pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")

CLUSTERS = r"""
#include "prepass.cuh"
using namespace zt::tcb;
static float x[1];
static __half planes[1];
static uint2 part[1];
static uint32_t amax[1];
static void add(PassArgs &a, int rows, int group) { pass_add(a, x, 1, rows, group, group, part, amax, nullptr, planes); }
int main() {
    long long taken = 0, refused = 0, bad = 0;
    const int rows[] = {1, 31, 64, 100, 127, 128, 129, 300, 512, 513, 1000, 1300, 2048, 4097}, groups[] = {1, 2, 3, 8, 17, 64};
    for (int units : {32, 64, 128, 160, 256, 512, 1024})
        for (int r0 : rows)
            for (int g0 : groups)
                for (int r1 : rows)
                    for (int g1 : groups) {
                        PassArgs a{};
                        a.dim = a.pd = 64;
                        add(a, r0, g0), add(a, r1, g1);
                        const long long c = pass_one_blocks(a, units);
                        (c ? taken : refused) += 1;
                        for (int i = 0; c && i < a.n; ++i) {
                            const long long n = (long long)a.t[i].rows * a.t[i].group;
                            if (n > c * units || n <= (c - 1) * units) {  // not all of it, or not a unit for the last block
                                if (bad++ < 5) printf("%d x %d and %d x %d, %d units a block: %lld blocks\n", r0, g0, r1, g1, units, c);
                            }
                        }
                    }
    for (int sms : {1, 2, 148, 160})
        for (long long steps = 1; steps <= kBackSteps; ++steps)
            for (long long bg = 1; bg <= 400; ++bg) {
                const PassBackPlan p = pass_backward_plan(steps, bg, sms);
                if (p.cluster < 1 || p.cluster > kOneCluster || p.per > 8 || (long long)p.cluster * p.per < steps || (long long)(p.cluster - 1) * p.per >= steps) {
                    if (bad++ < 5) printf("%lld steps, %lld groups, %d SMs: %d blocks of %d\n", steps, bg, sms, p.cluster, p.per);
                }
            }
    printf("%lld taken, %lld refused, %lld bad\n", taken, refused, bad);
    return bad > 0 || taken < 1000 || refused < 1000;
}
"""


def run(tmp_path, program):
    src = tmp_path / "program.cu"
    src.write_text(program)
    exe = str(tmp_path / "program")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", exe, str(src)])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_every_block_of_a_cluster_has_work(tmp_path):
    run(tmp_path, CLUSTERS)
