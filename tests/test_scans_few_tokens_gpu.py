"""The scans on states at any address, and on steps of few tokens: a request cut into steps of one to four tokens gives the
bits of the request in one step, whatever kernel the step's lengths choose."""
import pytest
import torch

from test_zesapel_gpu import batch_of, randn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIZES = [(1, 1), (8, 2), (9, 3), (16, 4), (17, 7), (32, 66), (33, 5), (64, 64), (65, 12), (128, 33), (129, 8), (256, 6)]


@pytest.fixture(scope="module")
def ops():
    from dlm_b200.ops import native_ops
    return native_ops(fast=True)


def scans(ops, N, P, T, heads=3):
    """The four walks (and retention) as functions of (first token, end, batch, state)."""
    xbc, dt = randn(T, heads * P + 2 * N, seed=1), randn(T, heads, seed=2)
    bias, A_log, D = randn(heads, seed=3, std=0.5), randn(heads, seed=4, std=0.5), randn(heads, seed=5)
    q, k, v, z = (randn(T, heads * n, seed=7 + i) for i, n in enumerate((N, N, P, N)))
    dec, beta, fixed = randn(T, heads, seed=11), randn(T, heads, seed=12), torch.linspace(0.8, 0.99, heads, device=DEV)
    vkq = torch.cat([v, k, q], 1)
    proj, lw, a_bias = randn(T, 4 * heads * N, seed=14), randn(T, heads * N, seed=15), randn(heads * N, seed=16)
    scale = N ** -0.5
    out = {
        "ssm": lambda a, e, b, s: ops.ssm_scan(xbc[a:e], dt[a:e], bias, A_log, D, s, b, heads, P, N, 1),
        "ssm, silu": lambda a, e, b, s: ops.ssm_scan(xbc[a:e].clone(), dt[a:e], bias, A_log, D, s, b, heads, P, N, 1,
                                                     silu_inputs=True),
        "retention": lambda a, e, b, s: ops.ssm_scan(vkq[a:e], None, None, None, None, s, b, heads, P, N, heads,
                                                     fixed_decay=fixed),
        "channel": lambda a, e, b, s: ops.gated_scan(q[a:e], k[a:e], v[a:e], z[a:e], None, s, b, heads, heads, N, P,
                                                     q_scale=scale, tau=8.0),
        "delta": lambda a, e, b, s: ops.gated_scan(q[a:e], k[a:e], v[a:e], dec[a:e], beta[a:e], s, b, heads, heads, N, P,
                                                   unit_eps=1e-6, q_scale=scale, A_log=A_log, decay_bias=bias),
    }
    if N == P:
        HN = heads * N
        out["removal"] = lambda a, e, b, s: ops.delta_scan(proj[a:e], (0, HN, 2 * HN, 3 * HN), lw[a:e], a_bias, s, b, heads, N,
                                                           1e-6, 0.6)
    return out


@pytest.mark.parametrize("N,P", [(16, 4), (64, 64), (128, 36), (24, 6)])
def test_a_state_may_lie_at_any_address(ops, N, P):
    """States at storage offsets that are no multiple of 16 bytes (shifted by one number) give what an aligned one gives."""
    heads, lens = 3, [21, 1, 6]
    b = batch_of(lens, [2, 0, 3])
    for name, run in scans(ops, N, P, sum(lens), heads).items():
        state = randn(5, heads, N, P, seed=6, std=0.3)
        shifted = torch.empty(state.numel() + 1, device=DEV)[1:].view(state.shape)
        shifted.copy_(state)
        want, got = run(0, sum(lens), b, state), run(0, sum(lens), b, shifted)
        assert torch.equal(got, want) and torch.equal(shifted, state), name
    ops.check_errors()


def cut(T):
    """``[(first, end), ...]``: steps of one, two, three, four, one, ... tokens, and one of six in the middle."""
    out, at, n = [], 0, 0
    while at < T:
        step = min([1, 2, 3, 4, 1, 6][n % 6], T - at)
        out.append((at, at + step))
        at, n = at + step, n + 1
    return out


@pytest.mark.parametrize("N,P", SIZES)
def test_few_tokens_give_the_same_bits(ops, N, P):
    heads, lens, slots = 3, [21, 1, 18], [2, 0, 3]
    starts = [0, 21, 22]
    for name, run in scans(ops, N, P, sum(lens), heads).items():
        first = randn(5, heads, N, P, seed=6, std=0.3)
        whole_state, cut_state = first.clone(), first.clone()
        whole = run(0, sum(lens), batch_of(lens, slots), whole_state)
        for n, s, slot in zip(lens, starts, slots):
            for a, e in cut(n):
                got = run(s + a, s + e, batch_of([e - a], [slot]), cut_state)
                assert torch.equal(got, whole[s + a:s + e]), (name, a, e)
        assert torch.equal(cut_state, whole_state), name
        # several short requests in one step
        together, alone = first.clone(), first.clone()
        both = run(0, 8, batch_of([3, 1, 4], [1, 4, 0]), together)
        for a, e, slot in ((0, 3, 1), (3, 4, 4), (4, 8, 0)):
            assert torch.equal(run(a, e, batch_of([e - a], [slot]), alone), both[a:e]), name
        assert torch.equal(together, alone), name
    ops.check_errors()


@pytest.mark.parametrize("inner,N", [(4, 1), (36, 8), (33, 9), (64, 16), (7, 33), (20, 256), (130, 12)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_selective_scan_of_few_tokens_gives_the_same_bits(ops, inner, N, dtype):
    lens, slots, starts = [21, 1, 18], [2, 0, 3], [0, 21, 22]
    T = sum(lens)
    x, dt, z, bc = randn(T, inner, seed=1), randn(T, inner, seed=2), randn(T, inner, seed=3), randn(T, 2 * N, seed=4)
    bias, A_log, D = randn(inner, seed=5), randn(inner, N, seed=6, std=0.5), randn(inner, seed=7)

    def run(a, e, b, s):
        return ops.selective_scan(x[a:e], dt[a:e], bc[a:e], z[a:e], bias, A_log, D, s, b, dtype)

    first = randn(5, inner, N, seed=8, std=0.3)
    whole_state, cut_state = first.clone(), first.clone()
    whole = run(0, T, batch_of(lens, slots), whole_state)
    for n, s, slot in zip(lens, starts, slots):
        for a, e in cut(n):
            got = run(s + a, s + e, batch_of([e - a], [slot]), cut_state)
            assert torch.equal(got, whole[s + a:s + e]), (a, e)
    assert torch.equal(cut_state, whole_state)
    ops.check_errors()


def test_selective_scan_keeps_decays_below_the_normal_numbers(ops):
    """Decays of 2^-127 to 2^-140 on a state of 2^120 and more: what is left of it is a normal number."""
    inner, N = 32, 16
    powers = torch.linspace(-140, -100, inner * N, dtype=torch.float64).view(inner, N)
    A_log = torch.log(-powers * 0.6931471805599453).float().to(DEV)      # decay 2^power at a step size of one
    bias = torch.full((inner,), 0.5413248546 - 1.0, device=DEV)         # softplus(ln(e - 1)) = 1
    for tokens in (1, 6):                                               # the kernel without a ring and the one with it
        dt = torch.full((tokens, inner), -60.0, device=DEV)             # the tokens after the first leave the state as it is
        dt[0] = 1.0
        zero, none = torch.zeros(tokens, inner, device=DEV), torch.zeros(inner, device=DEV)
        s = torch.full((1, inner, N), 2.0 ** 120, device=DEV)
        ops.selective_scan(zero, dt, torch.zeros(tokens, 2 * N, device=DEV), zero, bias, A_log, none, s, batch_of([tokens], [0]),
                           torch.float32)
        step = torch.nn.functional.softplus((dt[0] + bias).double().cpu())[:, None]
        want = 2.0 ** 120 * torch.exp(-step * torch.exp(A_log.double().cpu()))
        # an argument of 140 carries 2^-24 of itself, some 1e-5 of the decay; a decay of 2^-140 keeps nine bits
        assert torch.allclose(s[0].double().cpu(), want, rtol=4e-3)


def test_removal_with_short_keys_and_no_floor(ops):
    """Keys of length 1e-20: their square is no normal number and its reciprocal out of range, their unit vector is fine."""
    heads, d, lens = 2, 16, [7, 1]
    T, b = 8, batch_of([7, 1], [0, 1])
    proj, lw, a_bias = randn(T, 4 * heads * d, seed=1), randn(T, heads * d, seed=2), randn(heads * d, seed=3)
    HD = heads * d
    k = proj[:, HD:2 * HD]
    small = proj.clone()
    small[:, HD:2 * HD] = k * 2.0 ** -62       # |k|^2 about 2^-120
    small[:, 2 * HD:3 * HD] = proj[:, 2 * HD:3 * HD] * 2.0 ** 62
    tiny = proj.clone()
    tiny[:, HD:2 * HD] = k * 2.0 ** -67        # |k|^2 about 2^-130, its reciprocal beyond the largest number
    tiny[:, 2 * HD:3 * HD] = proj[:, 2 * HD:3 * HD] * 2.0 ** 67
    outs = []
    for p in (proj, small, tiny):
        s = randn(2, heads, d, d, seed=4, std=0.3)
        outs.append((ops.delta_scan(p, (0, HD, 2 * HD, 3 * HD), lw, a_bias, s, b, heads, d, 0.0, 0.6), s))
    for o, s in outs[1:]:
        # k v^T is as before and so is the unit vector, up to the bits that |k|^2 = 2^-130 keeps (about 19 of 24)
        assert torch.allclose(o, outs[0][0], atol=1e-3, rtol=1e-3) and torch.allclose(s, outs[0][1], atol=1e-3, rtol=1e-3)
