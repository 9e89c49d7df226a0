"""Rules of the kernel sources that no run can be trusted to show."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "z-transformer_b200", "csrc")


def sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def block(text, start):
    """The brace-balanced body that opens after `start`."""
    depth, i = 0, text.index("{", start)
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced")


def kernels():
    for name, text in sources().items():
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(([^;{]*?)\)\s*\{", text):
            yield name, m[1], m[2], block(text, m.start())


def test_overlapped_kernels_read_their_predecessors_results_with_plain_loads():
    """A kernel that calls pdl_wait() is resident while the launch before it still writes.  Loads through the read-only path
    may be moved ahead of the wait, so such kernels take no const __restrict__ pointer, and __ldg only reads what is at
    least two launches old: the caller's tensors, the rope table, kept planes, and in the attention kernels that have both launches
    of the pre-pass before them the first launch's row sums.  Up to 64 columns a backward's pre-pass may be one launch
    (pass_backward_kernel): there the row sums come from the launch just before."""
    overlapped = [(f, name, args, body) for f, name, args, body in kernels() if "pdl_wait()" in body]
    assert len(overlapped) >= 12
    older = {"reinterpret_cast<const uint2 *>(src", "reinterpret_cast<const float4 *>(t.x + at[k] * a.dim", "src + ch", "src + h4 + ch",
             "cs", "cs + 1", "p.lse", "p.delta", "p.rnorm"}
    for f, name, args, body in overlapped:
        assert not re.search(r"const [\w ]*\*\s*__restrict__", args), name
        for operand in re.findall(r"__ldg\(((?:[^()]|\([^()]*\))*)", body):
            assert any(operand.strip().startswith(o) for o in older), (name, operand)
        if f == "tc_bwd_fused64.cuh":
            assert not re.search(r"__ldg\(p\.(?:delta|rnorm)", body), name
        if f == "prepass.cuh":
            assert "__ldg(p.rnorm" not in body and "__ldg(t.rnorm" not in body, name
    # helpers of these kernels: V's planes come from the launch just before, and what a pre-pass of one launch reads may too
    assert "__ldg" not in block(sources()["prepass.cuh"], sources()["prepass.cuh"].index("void pass_held("))
    assert "__ldg" not in block(sources()["tc_bwd.cuh"], sources()["tc_bwd.cuh"].index("void row_to_tmem16("))


def test_aligned_cluster_barriers_are_reached_by_whole_warps():
    """barrier.cluster.*.aligned wants all threads of a warp to execute it together; code before it may end in one thread."""
    n = 0
    for name, text in sources().items():
        for m in re.finditer(r"barrier\.cluster\.(?:arrive|wait)[.\w]*\.aligned", text):
            body = text[text.rindex("__device__", 0, m.start()):m.start()]
            assert "__syncwarp();" in body, (name, m[0])
            n += 1
    assert n == 2


def test_aligned_tensor_memory_instructions_are_reached_by_whole_warps():
    """tcgen05.alloc, dealloc, ld, st and their waits are .sync.aligned: all threads of a warp execute them together.  They follow
    code that ends lane by lane (rows past the sequence, columns past the head, one lane's arrival), so the wrapper
    brings the warp together itself, and nothing but the wrappers issues them; a wait comes straight after the ones it is for or a
    vote of the whole warp.  A wrapper that does not (_joined) is called behind a vote, with no branch of a lane's own in between."""
    text = sources()
    names, joined = [], []
    for name, t in text.items():
        for m in re.finditer(r"tcgen05\.(?:alloc|dealloc|ld|st)[.\w:]*\.sync\.aligned", t):
            assert name == "tc_common.cuh", name
            start = t.rindex("__device__", 0, m.start())
            names.append(re.match(r"__device__ __forceinline__ void (\w+)\(", t[start:])[1])
            if names[-1].endswith("_joined"):
                joined.append(names[-1])
                continue
            body = t[start:m.start()]
            assert re.match(r"[^{]*\{\s*__syncwarp\(\);", body), names[-1]
    assert sorted(n.removesuffix("_joined") for n in names) == ["tmem_alloc", "tmem_dealloc", "tmem_ld16", "tmem_ld32", "tmem_st16", "tmem_st32", "tmem_st8"]
    for n in joined:
        assert re.search(r"void %s\([^{]*\{\s*__syncwarp\(\);\s*%s\(taddr, r\);" % (n.removesuffix("_joined"), n), text["tc_common.cuh"]), n
    uniform = {"if (diag)", "for (int c = 0; c < D; c += 32)", "for (int i = 0; i < 32; ++i)"}
    calls = 0
    for name, t in text.items():
        if name == "tc_common.cuh":
            continue
        for m in re.finditer(r"tmem_\w+_joined\(", t):
            calls += 1
            vote = max(t.rfind(x, 0, m.start()) for x in ("__all_sync(", "__any_sync(", "__syncwarp();"))
            between = t[t.index("\n", vote):m.start()]
            between = re.sub(r"//[^\n]*", "", between)
            branches = re.findall(r"\b(?:if|for|while|switch) \([^\n]*?\)(?= |$)", between, re.M)
            assert set(branches) <= uniform and "break" not in between.split("}", 1)[-1], (name, branches)
    assert calls == 24


def test_tensor_memory_is_allocated_before_the_next_launch_is_let_in():
    """A successor that is let in may take tensor memory of its own and then wait for this grid to end, so a block has its own by
    then: a barrier of the block lies between tmem_alloc and pdl_launch.  (A block without work, which returns, has none to wait for.)"""
    n = 0
    for f, name, args, body in kernels():
        if "tmem_alloc(" not in body or "pdl_launch();" not in body:
            continue
        n, body = n + 1, re.sub(r"//[^\n]*", "", body)
        for m in re.finditer(r"pdl_launch\(\);", body):
            depth, end = 1, m.end()  # of the braces that the call stands in
            while depth and end < len(body):
                depth += {"{": 1, "}": -1}.get(body[end], 0)
                end += 1
            if not body[m.end():end - 1].rstrip().endswith("return;") or end >= len(body):
                assert re.search(r"tmem_alloc\(.*__syncthreads\(\);", body[:m.start()], re.S), (f, name)
    assert n == 12
    # no other kernel has tensor memory, and none takes it in a function that this does not look into
    for name, text in sources().items():
        inside = sum(body.count("tmem_alloc(") for f, _, _, body in kernels() if f == name)
        assert text.count("tmem_alloc(") == inside + (name == "tc_common.cuh"), name


def test_rotated_query_rows_are_fenced_before_their_tile_is_copied_over():
    """rotate_q writes the query tile by ordinary stores, and bulk copies land there once a_ready has completed: an mbarrier's arrival
    orders no ordinary store before a bulk copy, so a proxy fence that runs wherever rows were rotated lies before it."""
    n = 0
    for name, text in sources().items():
        for m in re.finditer(r"(?<!void )rotate_q\(", text):
            n += 1
            end = text.index("mbar_arrive_warp(&sh->a_ready", m.end())
            if text.rfind("convert_q(uint8_t", 0, m.start()) > text.rfind("__global__", 0, m.start()):
                end = text.index("\n}\n", m.end())  # (its callers arrive)
            fences = re.findall(r"^ *(if \([^\n]*\) )?fence_async_smem\(\);", text[m.end():end], re.M)
            assert any(f in ("", "if (LO_SMEM || angles) ") for f in fences), name
    assert n == 3


def test_launches_go_under_their_kernels_names():
    """What a launch is recorded as (profiles, error messages) is the name of the kernel that runs."""
    n = 0
    defined = {name for _, name, _, _ in kernels()}
    for f, text in sources().items():
        for m in re.finditer(r"\blaunch_(?:pdl|pdl_cluster|after|pass_held)\(\"(\w+)\", (\w+)", text):
            n += 1
            if m[2] in defined:
                assert m[1] == m[2], (f, m[0])
            else:  # a variable: every kernel it may be has that name
                rest = text[m.end():].split("dim3")[0]
                picked = re.findall(r"\w+(?=<)", rest) if rest.startswith(" ?") else re.findall(r"\b%s = ([^;]*);" % m[2], text)
                assert picked and all(m[1] in x for x in picked), (f, m[0])
        for m in re.finditer(r"ZT_LAUNCH\(\"(\w+)\", \w+,\s*\((\w+)", text):
            n += 1
            assert m[1] == m[2], (f, m[0])
    assert n >= 20
