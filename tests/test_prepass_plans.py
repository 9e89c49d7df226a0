"""What the pre-passes' launches are planned to be (csrc/prepass.cuh, compiled here; without a device it takes a B200's 148 SMs): a cluster has a
unit, or a step, for each of its blocks, whichever tensor they convert; a unit's row, where it is taken by a product, is the division's."""
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

ROWS = r"""
#include "prepass.cuh"
using namespace zt::tcb;
int main() {
    long long products = 0, divisions = 0, bad = 0;
    const int groups[] = {1, 2, 3, 4, 5, 6, 7, 8, 12, 17, 31, 33, 64, 100, 511, 1000, 2000, 65535};
    for (int group : groups)
        // up to the longest that units are counted of in 31 bits, on both sides of where the product ends
        for (long long rows : {1ll, 2ll, 127ll, 1000ll, 65536ll, ((1ll << 32) / group - (1ll << 20)) / group - 1, ((1ll << 32) / group - (1ll << 20)) / group,
                               ((1ll << 32) / group - (1ll << 20)) / group + 1, 0x7fffffffll / group}) {
            if (rows < 1 || rows * group > 0x7fffffffll) continue;
            PassArgs a{};
            a.dim = a.pd = 32;
            static uint2 part[1];
            static uint32_t amax[1];
            const PassTensor &t = pass_add(a, nullptr, 1, (int)rows, group, group, part, amax, nullptr, nullptr);
            (t.per_head ? products : divisions) += 1;
            // a block's lanes ask for units beyond the last, as far as a step of all blocks: those only have to be beyond it, too
            const long long units = rows * group, step = (long long)t.slots * kPassThreads / 8 * kPassUnroll;
            for (long long r : {0ll, 1ll, 2ll, rows / 3, rows / 2, rows - 2, rows - 1})
                for (long long u : {r * group - 1, r * group, r * group + 1, r * group + group - 1})
                    if (u >= 0 && u < units && pass_row(t, (int)u) != u / group && bad++ < 5) printf("%lld x %d: unit %lld\n", rows, group, u);
            for (long long u : {units, units + 1, units + step - 1})
                if (u <= 0x7fffffffll && pass_row(t, (int)u) < rows && bad++ < 5) printf("%lld x %d: unit %lld, beyond\n", rows, group, u);
        }
    printf("%lld products, %lld divisions, %lld bad\n", products, divisions, bad);
    return bad > 0 || products < 40 || divisions < 10;
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


def test_a_units_row_is_the_divisions(tmp_path):
    run(tmp_path, ROWS)
