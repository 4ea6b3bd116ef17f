"""Convolutions in runs of tokens and norms of heads a warp, at the sizes where they take over: against the kernels for any
address (inputs shifted by one number take those) and the plain statement."""
import pytest
import torch

from plain_ops import PlainOps
from test_zesapel_gpu import batch_of, randn, to_cpu

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from dlm_b200.ops import native_ops
    return native_ops(fast=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,lens", [(516, [70, 1, 1, 3, 600]), (4, [75001]), (2052, [1] * 120 + [90, 35]), (4096, [1] * 123),
                                    (2048, [64, 65, 18]), (300004, [66])])
def test_convolutions_in_runs(ops, C, lens, dtype):
    T, b = sum(lens), batch_of(lens, list(range(len(lens))))
    x, w, bias = randn(T, C, seed=1), randn(C, 4, seed=2), randn(C, seed=3)
    odd = torch.empty(T, C + 4, device=DEV)[:, 1:C + 1]
    odd.copy_(x)
    for add, silu in ((False, True), (True, False)):
        one, two = (randn(len(lens), 3, C, seed=4) for _ in range(2))
        got, want = (ops.causal_conv(v, w, bias, s, b, add, silu, dtype) for v, s in ((x, one), (odd, two)))
        assert torch.equal(got, want) and torch.equal(one, two)


@pytest.mark.parametrize("T,gs,groups", [(1, 4, 7), (300, 132, 5), (257, 256, 2), (256, 256, 2), (19, 128, 3), (33, 64, 64)])
@pytest.mark.parametrize("mode", ["sigmoid_after", "silu_after"])
def test_norms_of_heads(ops, T, gs, groups, mode):
    y, gate, w = randn(T, groups * gs, seed=1), randn(T, groups * gs, seed=2), randn(groups * gs, seed=3)
    want = PlainOps().gated_rmsnorm(y.cpu(), gate.cpu(), w.cpu(), groups, 1e-5, mode, torch.float32)
    # sums of at most 256 squares in another order, then three products
    assert torch.allclose(ops.gated_rmsnorm(y, gate, w, groups, 1e-5, mode, torch.float32).cpu(), want, atol=2e-5, rtol=2e-5)


@pytest.mark.parametrize("d", [1, 9, 17, 33, 65, 129, 256, 257])
def test_removal_form_around_the_row_lanes(ops, d):
    """As the other scans' edges: 32-bit sums of at most d products of numbers around one, 41 tokens long."""
    heads, lens = 2, [41, 1, 18]
    T, HD, b = 60, 2 * d, batch_of([41, 1, 18], [2, 0, 3])
    proj, lw, a_bias = randn(T, 4 * HD, seed=1), randn(T, HD, seed=2), randn(HD, seed=3)
    state = randn(5, heads, d, d, seed=4, std=0.3)
    ws = state.clone().cpu()
    at = (0, HD, 2 * HD, 3 * HD)
    want = PlainOps().delta_scan(proj.cpu(), at, lw.cpu(), a_bias.cpu(), ws, to_cpu(b), heads, d, 1e-6, 0.6)
    got = ops.delta_scan(proj, at, lw, a_bias, state, b, heads, d, 1e-6, 0.6)
    assert torch.allclose(got.cpu(), want, atol=3e-4, rtol=3e-4) and torch.allclose(state.cpu(), ws, atol=3e-4, rtol=3e-4)
