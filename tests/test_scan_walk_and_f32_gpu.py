"""The register-tiled scans, the 32-bit tiles and the many-row latent attention at the edges of their tiles: sizes around
every number of row lanes, odd columns, rows around the row tiles, tokens around the runs a block takes."""
import math

import pytest
import torch

from plain_ops import PlainOps
from test_kernels_gpu import build_paged
from test_zesapel_gpu import _latent_case, _run_latent, batch_of, randn, to_cpu

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from dlm_b200.ops import native_ops
    return native_ops(fast=True)


@pytest.fixture(scope="module")
def slow_ops():
    from dlm_b200.ops import native_ops
    return native_ops(fast=False)


@pytest.mark.parametrize("N,P", [(1, 1), (8, 2), (9, 3), (16, 4), (17, 7), (32, 66), (33, 5), (64, 64), (65, 12), (128, 33),
                                 (129, 8), (256, 6), (257, 4)])
def test_scans_around_the_row_lanes(ops, N, P):
    """Sums of at most N products of numbers around one, 41 tokens long: 32-bit sums in another order differ by
    some sqrt(41 N) 2^-24 of their size."""
    heads, lens = 3, [41, 1, 18]
    T = sum(lens)
    ref, b = PlainOps(), batch_of(lens, [2, 0, 3])
    close = dict(atol=3e-4, rtol=3e-4)
    xbc, dt = randn(T, heads * P + 2 * N, seed=1), randn(T, heads, seed=2)
    bias, A_log, D = randn(heads, seed=3, std=0.5), randn(heads, seed=4, std=0.5), randn(heads, seed=5)
    state = randn(5, heads, N, P, seed=6, std=0.3)
    want_state = state.clone().cpu()
    want = ref.ssm_scan(xbc.cpu(), dt.cpu(), bias.cpu(), A_log.cpu(), D.cpu(), want_state, to_cpu(b), heads, P, N, 1)
    got = ops.ssm_scan(xbc, dt, bias, A_log, D, state, b, heads, P, N, 1)
    assert torch.allclose(got.cpu(), want, **close) and torch.allclose(state.cpu(), want_state, **close)
    q, k, v, z = (randn(T, heads * n, seed=7 + i) for i, n in enumerate((N, N, P, N)))
    dec, beta = randn(T, heads, seed=11), randn(T, heads, seed=12)
    for delta in (False, True):
        s = randn(5, heads, N, P, seed=13, std=0.3)
        ws = s.clone().cpu()
        if delta:
            kw = dict(unit_eps=1e-6, q_scale=N ** -0.5, A_log=A_log, decay_bias=bias)
            a = (q, k, v, dec, beta)
        else:
            kw = dict(q_scale=N ** -0.5, tau=8.0)
            a = (q, k, v, z, None)
        cpu = lambda t: t.cpu() if torch.is_tensor(t) else t
        want = ref.gated_scan(*map(cpu, a), ws, to_cpu(b), heads, heads, N, P, **{n: cpu(t) for n, t in kw.items()})
        got = ops.gated_scan(*a, s, b, heads, heads, N, P, **kw)
        assert torch.allclose(got.cpu(), want, **close) and torch.allclose(s.cpu(), ws, **close)
    ops.check_errors()


@pytest.mark.parametrize("N,K", [(16, 128), (17, 132), (130, 68), (258, 1412), (2048, 512)])
def test_32_bit_products_give_a_row_the_same_bits_in_every_batch(slow_ops, N, K):
    """One chain over k whatever the kernel: rows alone, in the kernels for few rows, in either tile, and as an expert's."""
    a, w, bias = randn(700, K, seed=1), randn(N, K, seed=2, std=0.05), randn(N, seed=3)
    whole = slow_ops.linear(a, w, bias, torch.float32)
    want = (a.double() @ w.double().T + bias.double()).float()
    assert torch.allclose(whole, want, rtol=2e-5, atol=2e-5 * math.sqrt(K))
    for first, n in ((0, 1), (5, 4), (0, 8), (3, 9), (1, 17), (0, 33), (0, 64), (0, 65), (100, 130)):
        assert torch.equal(slow_ops.linear(a[first:first + n], w, bias, torch.float32), whole[first:first + n])
    plain = slow_ops.linear(a, w, None, torch.float32)
    for sizes in ([0, 1, 9, 33, 70, 0, 5], [0] * 30 + [2, 1, 0, 3], [300, 0, 200]):
        off = torch.tensor([0] + torch.tensor(sizes).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
        n = int(off[-1])
        got = slow_ops.grouped_linear(a[:n], torch.stack([w * (1 + e % 3) for e in range(len(sizes))]), off)
        for e in range(len(sizes)):
            r0, r1 = int(off[e]), int(off[e + 1])
            if e % 3 == 0:
                assert torch.equal(got[r0:r1], plain[r0:r1])
            assert torch.allclose(got[r0:r1], plain[r0:r1] * (1 + e % 3), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("nh,nkv,hd", [(2, 1, 4), (4, 2, 64), (16, 16, 68), (40, 8, 128)])
def test_32_bit_attention_in_either_block(slow_ops, nh, nkv, hd):
    """Blocks of 16 queries (few heads and tokens) and of 32 (many): a query's bits do not depend on which it was in."""
    reqs = [(700, 513), (90, 1), (33, 33)]
    k, v, table, cu_q, kv_len = build_paged(reqs, nkv, hd, 16, torch.float32, 5)
    T = int(cu_q[-1])
    q = randn(T, nh * hd, seed=6)
    for window in (0, 50):
        whole = slow_ops.attention(q, k, v, table, cu_q, kv_len, window, hd ** -0.5, nh, nkv, hd, 513, 700, 1)
        want = PlainOps().attention(q, k, v, table, cu_q, kv_len, window, hd ** -0.5, nh, nkv, hd, 513, 700)
        assert torch.allclose(whole, want, rtol=1e-4, atol=2e-5)
        one = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
        for t in (0, 31, 32, 511, 512):
            n = torch.tensor([700 - 513 + t + 1], dtype=torch.int32, device=DEV)
            alone = slow_ops.attention(q[t:t + 1], k, v, table[:1], one, n, window, hd ** -0.5, nh, nkv, hd, 1, 700, 1)
            assert torch.equal(alone[0], whole[t])
    slow_ops.check_errors()


@pytest.mark.parametrize("H,rank,dr,window", [(16, 128, 8, 0), (8, 256, 64, 70), (20, 512, 64, 33), (3, 384, 0, 0),
                                              (4, 512, 512, 0)])
def test_latent_attention_of_many_rows(ops, H, rank, dr, window):
    """Enough tokens for the kernel whose blocks take 64 rows: requests that end inside a run, begin in the middle of a
    page, and hold less than a run, against the plain statement (bfloat16 latents).  The last rows are too long for it."""
    c = _latent_case(ops, torch.bfloat16, H, 16, dr, 8, rank, window, 16, lens=[301, 2, 333, 7], starts=[5, 40, 0, 77],
                     seed=rank, rot_dims=min(dr, 8))
    got, want = _run_latent(ops, c)
    assert torch.allclose(got, want, atol=3e-2, rtol=3e-2)
    ops.check_errors()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,lens", [(4, [65]), (516, [70, 1, 1, 3, 64]), (2048, [2, 301, 1]), (6, [90])])
def test_causal_convolution_in_runs(ops, dtype, C, lens):
    """Runs of tokens that end inside a request, begin at one, and hold several; an odd channel count keeps the other kernel."""
    T, b = sum(lens), batch_of(lens, list(range(len(lens))))
    x, w, bias = randn(T, C + 4, seed=1)[:, :C], randn(C, 4, seed=2), randn(C, seed=3)
    for add, silu in ((False, True), (True, False)):
        state = randn(len(lens) + 1, 3, C, seed=4)
        ws = state.clone().cpu()
        want = PlainOps().causal_conv(x.cpu(), w.cpu(), bias.cpu(), ws, to_cpu(b), add, silu, dtype)
        got = ops.causal_conv(x, w, bias, state, b, add, silu, dtype)
        close = dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=1e-2, rtol=1e-2)
        assert torch.allclose(got.cpu().float(), want.float(), **close) and torch.equal(state.cpu(), ws)


@pytest.mark.parametrize("inner,N", [(4, 1), (36, 8), (33, 9), (64, 16), (7, 33), (20, 256)])
def test_selective_scan_around_the_state_lanes(ops, inner, N):
    lens = [41, 1, 18]
    T, b = sum(lens), batch_of(lens, [2, 0, 3])
    x, dt, z, bc = randn(T, inner, seed=1), randn(T, inner, seed=2), randn(T, inner, seed=3), randn(T, 2 * N, seed=4)
    bias, A_log, D = randn(inner, seed=5), randn(inner, N, seed=6, std=0.5), randn(inner, seed=7)
    state = randn(5, inner, N, seed=8, std=0.3)
    ws = state.clone().cpu()
    want = PlainOps().selective_scan(x.cpu(), dt.cpu(), bc.cpu(), z.cpu(), bias.cpu(), A_log.cpu(), D.cpu(), ws, to_cpu(b),
                                     torch.float32)
    got = ops.selective_scan(x, dt, bc, z, bias, A_log, D, state, b, torch.float32)
    assert torch.allclose(got.cpu(), want, atol=3e-4, rtol=3e-4) and torch.allclose(state.cpu(), ws, atol=3e-4, rtol=3e-4)


@pytest.mark.parametrize("gs,groups", [(4, 7), (64, 32), (128, 3), (132, 5), (256, 2), (512, 1), (4096, 1)])
@pytest.mark.parametrize("mode", ["silu_before", "sigmoid_after", "silu_after"])
def test_gated_norm_of_heads_and_wide_rows(ops, gs, groups, mode):
    y, gate, w = randn(19, groups * gs, seed=1), randn(19, groups * gs, seed=2), randn(groups * gs, seed=3)
    want = PlainOps().gated_rmsnorm(y.cpu(), gate.cpu(), w.cpu(), groups, 1e-5, mode, torch.float32)
    assert torch.allclose(ops.gated_rmsnorm(y, gate, w, groups, 1e-5, mode, torch.float32).cpu(), want, atol=2e-5, rtol=2e-5)
