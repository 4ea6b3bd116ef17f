"""The rule that kernels launched with programmatic dependent launch keep (``dep_wait`` in common.cuh), read off their
sources: a race that it excludes shows on a device only now and then."""
import glob
import os
import re
import threading

import pytest

SOURCES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dlm_b200", "csrc", "kernels")


def kernels():
    """``(file, name, parameters, body)`` of every kernel that waits for the kernel before it; comments taken out."""
    out = []
    for path in sorted(glob.glob(os.path.join(SOURCES, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            head_end = text.index(") {\n", m.start())
            head, body = text[m.start():head_end], text[head_end:text.index("\n}\n", head_end)]
            if "dep_wait()" in body:
                head = re.sub(r"__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)", "", head)
                name = re.search(r"(\w+)\s*\(", head).group(1)
                out.append((os.path.basename(path), name, head[head.index(name) + len(name) + 1:], body))
    return out


KERNELS = kernels()


def test_the_kernels_were_found():
    names = {k[1] for k in KERNELS}
    assert {"gemm_tc_kernel", "gemm_tc_pair_kernel", "gemm_stream_kernel", "attention_prefill_tc_kernel",
            "rmsnorm_kernel", "causal_conv_runs_kernel"} <= names


@pytest.mark.parametrize("file,name,params,body", KERNELS, ids=[f"{k[0]}:{k[1]}" for k in KERNELS])
def test_nothing_is_looked_up_or_taken_before_the_wait(file, name, params, body):
    """Offsets of groups are an earlier kernel's output; tensor memory and a cluster's barrier are what another block may
    wait for."""
    before = body[:body.index("dep_wait()")]
    for word in ("tile_info", "expert_offsets[", "tcgen05.alloc", "cluster_sync_all"):
        assert word not in before, f"{name} uses {word} before it waits for the kernel before it"


@pytest.mark.parametrize("name", ["router_logits_multi_kernel", "router_fused_kernel"])
def test_a_router_that_reads_before_the_wait_reads_past_l1(name):
    (body,) = [k[3] for k in KERNELS if k[1] == name]
    assert "load_settled(" in body and not re.search(r"to_f32\((?:src|h)\[", body)


# weights, tables and constants, and what the host copies to the device before a step's first kernel
NO_KERNEL_WRITES = set("""w b w2 b2 wa wb w_post w_next norm_w qn_w kn_w kvn_w bias vec sink sinks slopes select_bias table added a mix
    outw in_next inv_freq tokens idx positions slots block_table cu_q kv_len token_req state_slot""".split())


@pytest.mark.parametrize("file,name,params,body", KERNELS, ids=[f"{k[0]}:{k[1]}" for k in KERNELS])
def test_what_kernels_write_is_not_declared_read_only(file, name, params, body):
    """A load through a ``__restrict__`` pointer to const may take the path for data that nothing writes while the kernel is
    resident, or move above the wait; so may ``__ldg``."""
    text = open(os.path.join(SOURCES, file)).read()
    launched_early = re.search(r"launch_dep\(\s*" + name + r"\b", text) or (
        re.search(r"launch_dep\(\s*kern\b", text) and re.search(r"kern = [^;]*\b" + name + r"\b", text))
    if launched_early:
        assert set(re.findall(r"__restrict__ (\w+)", params)) <= NO_KERNEL_WRITES
        assert set(re.findall(r"__ldg\([^;]*?(\w+) \+", body)) <= {"w4"}


def test_every_wait_on_a_barrier_is_bounded_in_time():
    """A loop of tries of its own is bounded in tries at best, and each try may block for a while; and a bound in time must not
    run while the kernel before this one does."""
    for path in glob.glob(os.path.join(SOURCES, "*.cu")):
        assert not re.search(r"(?:for|while) \([^\n]*\)[^;{]*\{?\s*(?:if \()?!?mbar_try_wait", open(path).read()), path
    (body,) = [k[3] for k in KERNELS if k[1] == "gemm_stream_kernel"]
    producer = body[body.index("if (warp == CW)"):]
    assert "dep_wait()" in producer[:producer.index("mbar_wait(&empty_bar")]
    (body,) = [k[3] for k in KERNELS if k[1] == "attention_decode_tma_kernel"]
    assert re.search(r"it >= NST\) && !waited\) \{ dep_wait\(\)", body[:body.index("mbar_wait(&empty_bar")])


def test_the_setting_belongs_to_a_thread():
    """Two engines in two threads, one of a design that asks for ordinary launches: neither changes the other's setting, and
    both find their own as it was whichever ends first."""
    from dlm_b200.build import load_kernels
    from dlm_b200.ops.native import NativeOps
    ops = NativeOps.__new__(NativeOps)
    ops.k = load_kernels()
    before = bool(ops.k.dep_launch_enabled())
    entered, leave, seen = threading.Event(), threading.Event(), []

    def other():
        ops.k.set_dep_launch(True)
        with ops.dependent_launch(False):
            entered.set()
            assert leave.wait(30)
            seen.append(bool(ops.k.dep_launch_enabled()))
        seen.append(bool(ops.k.dep_launch_enabled()))

    t = threading.Thread(target=other)
    try:
        ops.k.set_dep_launch(True)
        t.start()
        assert entered.wait(30)
        seen.append(bool(ops.k.dep_launch_enabled()))      # this thread's, while the other has it off
        with ops.dependent_launch(False):
            leave.set()
            t.join()
            seen.append(bool(ops.k.dep_launch_enabled()))  # the other has put its own back
        seen.append(bool(ops.k.dep_launch_enabled()))
    finally:
        leave.set()
        ops.k.set_dep_launch(before)
    assert seen == [True, False, True, False, True]
