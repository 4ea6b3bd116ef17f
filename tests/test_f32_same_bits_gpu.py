"""The 32-bit products and attention in register tiles against the kernels that take any address: the same bits.  Operands
shifted by one number (their rows cannot be fetched 16 bytes at a time) take the older kernel."""
import pytest
import torch

from test_kernels_gpu import build_paged
from test_zesapel_gpu import randn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from dlm_b200.ops import native_ops
    return native_ops(fast=False)


def shifted(t):
    """The same numbers, contiguous, at an address four bytes beyond a multiple of 16."""
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    out.copy_(t)
    return out


# rows on both sides of the few-row kernels' tiles and of the switch to the larger tiles, columns that are no multiple of a tile
@pytest.mark.parametrize("M,N,K", [(1, 16, 128), (7, 130, 68), (8, 258, 1412), (9, 258, 132), (16, 64, 64), (17, 34, 100),
                                   (32, 130, 260), (33, 130, 260), (64, 98, 36), (64, 10050, 64), (40, 16388, 20), (65, 9700, 48),
                                   (130, 9602, 36), (513, 2050, 68), (1030, 5122, 36), (700, 130, 64)])
def test_products(ops, M, N, K):
    a, w, bias = randn(M, K, seed=1), randn(N, K, seed=2, std=0.1), randn(N, seed=3)
    b = shifted(a)
    for act in (None, bias):
        assert torch.equal(ops.linear(a, w, act, torch.float32), ops.linear(b, w, act, torch.float32))
    one, two = randn(M, N, seed=4), randn(M, N, seed=4)
    ops.linear_add(a, w, one)
    ops.linear_add(b, w, two)
    assert torch.equal(one, two)
    assert torch.equal(ops.linear_swiglu(a, w), ops.linear_swiglu(b, w))
    assert torch.equal(ops.linear_act(a, w, "gelu"), ops.linear_act(b, w, "gelu"))


@pytest.mark.parametrize("sizes", [[0, 1, 9, 33, 70, 0, 5], [0] * 30 + [2, 1, 0, 3], [300, 0, 200], [16, 17, 15, 16], [5] * 40])
@pytest.mark.parametrize("N,K", [(130, 68), (2818, 36)])
def test_grouped_products(ops, sizes, N, K):
    off = torch.tensor([0] + torch.tensor(sizes).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    n = int(off[-1])
    a, w = randn(n, K, seed=1), randn(len(sizes), N, K, seed=2, std=0.1)
    assert torch.equal(ops.grouped_linear(a, w, off), ops.grouped_linear(shifted(a), w, off))
    rows = torch.randperm(n, generator=torch.Generator().manual_seed(5)).to(torch.int32).to(DEV)
    assert torch.equal(ops.grouped_swiglu(a, w, off, rows), ops.grouped_swiglu(shifted(a), w, off, rows))


@pytest.mark.parametrize("nh,nkv,hd", [(2, 1, 4), (4, 2, 16), (4, 2, 20), (4, 2, 64), (6, 6, 68), (40, 8, 128)])
def test_attention(ops, nh, nkv, hd):
    reqs = [(700, 213), (90, 1), (33, 33), (300, 2)]
    k, v, table, cu_q, kv_len = build_paged(reqs, nkv, hd, 16, torch.float32, 5)
    q = randn(int(cu_q[-1]), nh * hd, seed=6)
    sinks, slopes = randn(nh, seed=7), randn(nh, seed=8).abs() * 0.01
    forms = [dict(), dict(window=50), dict(window=50, keep_first=3), dict(chunk=64), dict(sinks=sinks), dict(slopes=slopes),
             dict(softcap=20.0), dict(parts=2)]
    for form in forms:
        form = dict(form)
        if form.get("parts") == 2 and (nh % 2 or hd % 2):
            continue
        window = form.pop("window", 0)
        x = q
        if form.get("parts") == 2:
            x = q.view(-1, nh, 2, hd // 2).clone()
            x[:, 0::2, 1] = 0
            x[:, 1::2, 0] = 0
            x = x.view(-1, nh * hd)
        got = [ops.attention(t, k, v, table, cu_q, kv_len, window, hd ** -0.5, nh, nkv, hd, 213, 700, 1, **form)
               for t in (x, shifted(x))]
        assert torch.equal(*got), form
    ops.check_errors()
