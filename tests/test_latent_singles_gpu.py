"""Requests of one token beside prompts in one step of the latent attention: taken apart (many keys) or not, with and without a
sink, against the plain statement; steps of prompts alone and of single tokens alone as they are."""
import pytest
import torch

from test_zesapel_gpu import _latent_case, _run_latent

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,rank,dr,window", [(16, 128, 8, 0), (8, 256, 64, 0), (20, 512, 64, 0), (16, 512, 64, 33)])
@pytest.mark.parametrize("lens,starts", [([1, 301, 1, 333, 1, 7, 1], [1500, 5, 0, 40, 40, 9, 700]), ([400], [1100]),
                                         ([1] * 40 + [500], [1030 + 3 * i for i in range(40)] + [0])])
def test_single_tokens_beside_prompts(H, rank, dr, window, lens, starts):
    from dlm_b200.ops import native_ops
    ops = native_ops(fast=True)
    c = _latent_case(ops, torch.bfloat16, H, 16, dr, 8, rank, window, 16, lens=lens, starts=starts, seed=rank, rot_dims=min(dr, 8))
    together, want = _run_latent(ops, c)
    assert torch.allclose(together, want, atol=3e-2, rtol=3e-2)
    c["b"].num_single, c["b"].max_kv_len = sum(n == 1 for n in lens), max(s + n for s, n in zip(starts, lens))
    apart, _ = _run_latent(ops, c)
    # bfloat16 results of the same 32-bit sums in another order
    assert torch.allclose(apart, want, atol=3e-2, rtol=3e-2) and torch.allclose(apart, together, atol=2e-2, rtol=2e-2)
    assert (apart - together).norm() < 4e-3 * together.norm()
    ops.check_errors()
