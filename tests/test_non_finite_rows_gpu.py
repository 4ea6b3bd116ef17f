"""A latent that is not finite reaches the tokens that see it and no other, whichever tokens share a block with them."""
import pytest
import torch

from test_zesapel_gpu import batch_of, randn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("window", [0, 33])
@pytest.mark.parametrize("H,rank,dr", [(16, 512, 64), (8, 256, 32), (3, 128, 8)])
def test_latent_attention(H, rank, dr, window, bad):
    from dlm_b200.ops import native_ops
    ops = native_ops(fast=True)
    T, page, at = 1201, 16, 150
    pages = -(-T // page)
    b = batch_of([T], [0])
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, pages)
    cache = randn(pages, 1, page, rank + dr, seed=1).to(torch.bfloat16)
    q_lat, q_rot = randn(H, T, rank, seed=2, std=0.2), randn(T, H, dr, seed=3, std=0.2)

    def run(c):
        return ops.latent_attention(q_lat, q_rot, None, c, table, b, H, dr, rank, window, 0.1).float()

    clean = run(cache)
    broken = cache.clone()
    broken[at // page, 0, at % page, 5] = bad
    got = run(broken)
    sees = torch.arange(T, device=DEV) >= at
    if window:
        sees &= torch.arange(T, device=DEV) < at + window
    assert not torch.isfinite(got[:, sees]).all(dim=-1).any()
    assert torch.isfinite(got[:, ~sees]).all()
    # (the rows of a run with such a key add the chunk's products up in another order)
    assert torch.allclose(got[:, ~sees], clean[:, ~sees], atol=1e-2, rtol=1e-2)
    ops.check_errors()
