"""The recurrent gated unit of long bfloat16 prompts (one grouped product for the gates, clusters for the recurrence) beside a
64-bit walk: lengths around a warp's, a block's and a round's tokens, convolutions of 1 to 8 taps over carried inputs, narrow
and wide diagonal blocks.

Bounds.  The gates' operand u is rounded to bfloat16 (2^-9 of each number, independent over a block's channels), and so are the
outputs: a row's outputs are off by about 2^-9 of its norm, bounded by 6e-3; states see the gates' rounding alone: 4e-3.  The
carried inputs are the projection's own numbers plus a bias: the bits of a 32-bit sum."""
import pytest
import torch

from test_piece_products_gpu import calls, close, plan_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,blocks,taps", [(256, 1, 4), (72, 3, 1), (320, 5, 8), (1056, 4, 3), (16, 2, 2)])
@pytest.mark.parametrize("news,starts", [([128], [0]), ([513, 1, 7], [0, 2, 300]), ([5, 1029], [1, 9])])
@pytest.mark.parametrize("pad", [0, 2])
def test_prompts(W, blocks, taps, news, starts, pad, monkeypatch):
    """``pad``: columns behind the projection's; with two of them its rows are off 16 bytes, and the passes over pieces take the step."""
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
    names = calls(k, monkeypatch)
    T, bs = plan.T, W // blocks
    g = torch.Generator(device="cuda").manual_seed(W + taps + T)

    def rand(*shape, scale=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * scale).bfloat16()
    proj = rand(T, 2 * W + pad)
    bx, by, cb, cr, ci, lam = (rand(W, scale=0.3) for _ in range(6))
    conv_w, ar, ai = rand(W, taps, scale=0.5), rand(blocks, bs, bs, scale=bs ** -0.5), rand(blocks, bs, bs, scale=bs ** -0.5)
    first = torch.randn((plan.R, taps, W), generator=g, device="cuda")
    for r, s in enumerate(starts):                    # (a sequence that starts here has a state of zeros)
        if s == 0:
            first[plan.R - 1 - r] = 0
    state, out = first.clone(), torch.full((T, W), float("nan"), device="cuda", dtype=torch.bfloat16)
    k.rglru(out, proj, W, 0, bx, by, conv_w, cb, ar, ai, cr, ci, lam, 8.0, state, plan, W, blocks, taps, 0.7,
            gates=torch.cat([ar, ai], dim=1).contiguous())
    assert ("zlm_rglru_cluster" in names, "zlm_rglru" in names) == (not pad, bool(pad))
    want, S = torch.empty((T, W), dtype=torch.float64, device="cuda"), first.double()
    gelu = torch.nn.functional.gelu(proj[:, :W].double() + by.double(), approximate="tanh")
    at = 0
    for r, n in enumerate(news):
        slot = plan.R - 1 - r
        before = S[slot, 1:].clone()
        if starts[r] < taps - 1:
            before[:taps - 1 - starts[r]] = 0         # positions ahead of the sequence's first count as zeros
        ext = torch.cat([before, (proj[at:at + n, W:2 * W].float() + bx.float()).double()])
        u = sum(ext[j:j + n] * conv_w[:, j].double() for j in range(taps)) + cb.double()
        ub = u.view(n, blocks, bs)
        rg, ig = (torch.sigmoid(torch.einsum("nbi,boi->nbo", ub, m.double()).flatten(1) + b.double()) for m, b in ((ar, cr), (ai, ci)))
        log_a = -8.0 * rg * torch.nn.functional.softplus(lam.double())
        a, b = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * ig * u
        s = S[slot, 0].clone()
        for t in range(n):
            s = a[t] * s + b[t]
            want[at + t] = s
        S[slot, 0] = s
        kept = torch.cat([S[slot, 1:], ext[taps - 1:]])
        S[slot, 1:] = kept[kept.shape[0] - (taps - 1):]
        at += n
    close(out, want * gelu * 0.7, 6e-3)
    close(state[:, 0], S[:, 0], 4e-3)
    assert torch.equal(state[:, 1:], S[:, 1:].float())


def _function(which, x):
    import ctypes

    from zlm_b200.kernels import get_kernels
    k, out = get_kernels(), torch.empty_like(x)
    k._call("zlm_rglru_functions", k._p(out), k._p(x), ctypes.c_int(x.numel()), ctypes.c_int(which), k._stream())
    return out


def _spread(lo, hi, n=20001):
    """``n`` numbers of [lo, hi], and as many spread over the logarithm towards zero, of either sign where the range has both."""
    x = torch.linspace(lo, hi, n, dtype=torch.float64)
    small = torch.pow(10.0, torch.linspace(-44, 0, n, dtype=torch.float64))
    x = torch.cat([x, small[small <= hi], -small[small <= -lo]])
    return x.float().cuda()


# Units in the last place are 2^-23 of a number at most.  The exponential is off by up to two of them, the reciprocal after its step
# by one, every product and sum by half: five for sigmoid; four for 1 - e^y (e^(y/2) twice over, of at most 0.6 of the result,
# or a Horner chain whose terms shrink); the approximate root by two, and by half for its product.
@pytest.mark.parametrize("which,lo,hi,ulps,want", [
    (0, -100.0, 100.0, 5, torch.sigmoid), (1, -200.0, 0.0, 4, lambda y: -torch.expm1(y)), (2, 0.0, 1.0, 3, torch.sqrt)])
def test_functions_to_the_last_places(which, lo, hi, ulps, want):
    x = _spread(lo, hi)
    x = torch.cat([x, torch.tensor([-1.0, -1.0 - 2.0 ** -23, -1.0 + 2.0 ** -24, 1e-30, 9.9e-31, 2.0 ** -126, 0.0], device="cuda").clamp(lo, hi)])
    got, exact = _function(which, x).double(), want(x.double())
    # (below 2^-126 a unit is 2^-149 whatever the number is)
    assert ((got - exact).abs() <= ulps * torch.clamp(exact.abs() * 2.0 ** -23, min=2.0 ** -149)).all()
    assert torch.isnan(_function(which, torch.tensor([float("nan")], device="cuda"))).all()


def test_gelu_over_the_whole_range():
    """z sigmoid(2 t), t = c (z + 0.044715 z^3): as sigmoid, and its argument's three roundings times its slope, |2 t| relative to
    the result where that is small; nothing is left of the tail, however large the number, and what is not finite is what
    0.5 z (1 + tanh t) makes of it."""
    z = _spread(-12.0, 12.0)
    got, x = _function(3, z).double(), z.double()
    t2 = 1.5957691216057308 * (x + 0.044715 * x ** 3)
    exact = x * torch.sigmoid(t2)
    assert ((got - exact).abs() <= (6 + 4 * t2.abs()) * 2.0 ** -23 * exact.abs() + 2.0 ** -149 * (1 + x.abs())).all()
    far = torch.tensor([-1e4, -1e13, -1e30, -3.3895e38, 1e13, 3.3895e38], device="cuda")
    assert torch.equal(_function(3, far), torch.where(far < 0, torch.zeros_like(far), far))
    edge = _function(3, torch.tensor([float("inf"), float("-inf"), float("nan")], device="cuda"))
    assert edge[0] == float("inf") and torch.isnan(edge[1:]).all()
    edge = _function(0, torch.tensor([float("inf"), float("-inf"), -200.0], device="cuda"))
    assert edge.tolist() == [1.0, 0.0, 0.0]


@pytest.mark.parametrize("taps", [1, 4, 8])
def test_every_cluster_size_gives_the_same_bits(taps, monkeypatch):
    """Sequences from one token to more than two rounds of the largest cluster, side by side: blocks without a token leave, and the
    blocks' parts are folded one after the other whatever shares them."""
    from zlm_b200.kernels import get_kernels
    k, W, blocks = get_kernels(), 96, 2
    news, starts = [1, 128, 2, 1100, 64, 65, 1, 513, 9], [5, 0, 1, 300, 0, 2, 0, 7, 40]
    plan, T, bs = plan_of(news, starts), sum(news), W // blocks
    g = torch.Generator(device="cuda").manual_seed(taps)

    def rand(*shape, scale=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * scale).bfloat16()
    proj, gates = rand(T, 2 * W), rand(blocks, 2 * bs, bs, scale=bs ** -0.5)
    bx, by, cb, cr, ci, lam = (rand(W, scale=0.3) for _ in range(6))
    conv_w, first = rand(W, taps, scale=0.5), torch.randn((plan.R, taps, W), generator=g, device="cuda")
    ar, ai = (gates[:, i * bs:(i + 1) * bs].contiguous() for i in (0, 1))
    results = []
    for size in (8, 4, 2, 1):
        monkeypatch.setattr(k.lib, "zlm_rglru_cluster_size", lambda *a: size)
        state, out = first.clone(), torch.full((T, W), float("nan"), device="cuda", dtype=torch.bfloat16)
        k.rglru(out, proj, W, 0, bx, by, conv_w, cb, ar, ai, cr, ci, lam, 8.0, state, plan, W, blocks, taps, gates=gates)
        results.append((out, state))
    assert not torch.isnan(results[0][0]).any()
    for out, state in results[1:]:
        assert torch.equal(out, results[0][0]) and torch.equal(state, results[0][1])
