"""The recurrent gated unit of long bfloat16 prompts (one grouped product for the gates, clusters for the recurrence) beside a
64-bit walk: lengths around a warp's, a block's and a round's tokens, convolutions of 1 to 8 taps over carried inputs, narrow
and wide diagonal blocks.

Bounds.  The gates' operand u is rounded to bfloat16 (2^-9 of each number, independent over a block's channels), and so are the
outputs: a row's outputs are off by about 2^-9 of its norm, bounded by 6e-3; states see the gates' rounding alone: 4e-3.  The
carried inputs are the projection's own numbers plus a bias: the bits of a 32-bit sum."""
import pytest
import torch

from test_piece_products_gpu import close, plan_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,blocks,taps", [(256, 1, 4), (72, 3, 1), (320, 5, 8), (1056, 4, 3), (16, 2, 2)])
@pytest.mark.parametrize("news,starts", [([128], [0]), ([513, 1, 7], [0, 2, 300]), ([5, 1029], [1, 9])])
def test_prompts(W, blocks, taps, news, starts):
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
    T, bs = plan.T, W // blocks
    g = torch.Generator(device="cuda").manual_seed(W + taps + T)

    def rand(*shape, scale=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * scale).bfloat16()
    proj = rand(T, 2 * W)
    bx, by, cb, cr, ci, lam = (rand(W, scale=0.3) for _ in range(6))
    conv_w, ar, ai = rand(W, taps, scale=0.5), rand(blocks, bs, bs, scale=bs ** -0.5), rand(blocks, bs, bs, scale=bs ** -0.5)
    first = torch.randn((plan.R, taps, W), generator=g, device="cuda")
    for r, s in enumerate(starts):                    # (a sequence that starts here has a state of zeros)
        if s == 0:
            first[plan.R - 1 - r] = 0
    state, out = first.clone(), torch.full((T, W), float("nan"), device="cuda", dtype=torch.bfloat16)
    k.rglru(out, proj, W, 0, bx, by, conv_w, cb, ar, ai, cr, ci, lam, 8.0, state, plan, W, blocks, taps, 0.7,
            gates=torch.cat([ar, ai], dim=1).contiguous())
    want, S = torch.empty((T, W), dtype=torch.float64, device="cuda"), first.double()
    gelu = torch.nn.functional.gelu(proj[:, :W].double() + by.double(), approximate="tanh")
    at = 0
    for r, n in enumerate(news):
        slot = plan.R - 1 - r
        before = S[slot, 1:].clone()
        if starts[r] < taps - 1:
            before[:taps - 1 - starts[r]] = 0         # positions ahead of the sequence's first count as zeros
        ext = torch.cat([before, (proj[at:at + n, W:].float() + bx.float()).double()])
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
