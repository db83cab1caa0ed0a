"""Linear attention with decays per channel or per head over prompts in pieces, alone and with the heads' norm and gate, beside
a 64-bit walk: lengths around a piece's edges, key widths around the kernels' 32, 64 and 128 rows, value widths that are no
multiple of four or wider than a block, states carried in.

Bounds.  Sums of some ten to hundred fp32 products, 2^-24 of each: 1e-6 of the norm; gated outputs are rounded to their type."""
import pytest
import torch

from test_piece_products_gpu import calls, close, plan_of, unit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,D,V", [(2, 64, 128), (3, 20, 72), (1, 128, 30), (2, 33, 136)])
@pytest.mark.parametrize("news,starts", [([128], [0]), ([129, 1, 33], [0, 5, 300]), ([31, 200], [9, 0])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("per_head", [False, True])
def test_pieces(H, D, V, news, starts, dtype, per_head, monkeypatch):
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
    T = plan.T
    gen = torch.Generator(device="cuda").manual_seed(D + V + T)
    proj = torch.randn((T, 2 * H * D + 2 * H * V + 3), generator=gen, device="cuda").to(dtype)
    # decays from almost nothing kept to almost everything
    alpha = torch.sigmoid(torch.randn((T, H * D), generator=gen, device="cuda") * 4)
    head = torch.linspace(0.5, 0.99, H, device="cuda")
    first = torch.randn((plan.R, H, D, V), generator=gen, device="cuda")
    q, key = (proj[:, i * H * D:(i + 1) * H * D].double().view(T, H, D) for i in (0, 1))
    v = proj[:, 2 * H * D:2 * H * D + H * V].double().view(T, H, V)
    a = head.double()[:, None].expand(T, H, D) if per_head else alpha.double().view(T, H, D)
    want, S = torch.empty((T, H, V), dtype=torch.float64, device="cuda"), first.double()
    at = 0
    for r, n in enumerate(news):
        s = S[plan.R - 1 - r]
        for t in range(at, at + n):
            s = a[t][:, :, None] * s + key[t][:, :, None] * v[t][:, None]
            want[t] = (s * q[t][:, :, None]).sum(1) * 0.3
        S[plan.R - 1 - r] = s
        at += n
    args = (proj, 0, H * D, 2 * H * D, None if per_head else alpha, head if per_head else None)
    state, o = first.clone(), torch.full((T, H * V), float("nan"), device="cuda")
    k.linear_attention(o, *args, state, plan, H, D, V, 0.3)
    close(o, want.flatten(1), 1e-6)
    close(state, S, 1e-6)
    gate, w = proj[:, 2 * H * D + H * V:2 * H * D + 2 * H * V], torch.rand((V,), generator=gen, device="cuda") + 0.5
    state, y = first.clone(), torch.full((T, H * V), float("nan"), device="cuda", dtype=dtype)
    names = calls(k, monkeypatch)
    k.linear_attention_gated(y, gate, w, 1e-6, "silu", o, *args, state, plan, H, D, V, 0.3)
    assert names == ["zlm_linear_attention"] + ["zlm_norm_gate"] * (V > 128)
    z = gate.double()
    close(y, (unit(want) * w.double()).flatten(1) * z * torch.sigmoid(z), 4e-3 if dtype == torch.bfloat16 else 2e-6)
    close(state, S, 1e-6)


def test_heads_of_more_columns_than_a_grid_numbers():
    """A head of 600,008 value columns over 64 rows: the chain of its pieces would have 75,001 blocks, so its tokens are walked.  Columns
    know nothing of each other: its first and last ones are those of narrow heads walked alike, to the bit."""
    from zlm_b200.kernels import get_kernels
    k, T, D, V, n = get_kernels(), 128, 64, 600_008, 136
    g = torch.Generator(device="cuda").manual_seed(3)
    qk, v = (torch.randn((T, w), generator=g, device="cuda").bfloat16() for w in (2 * D, V))
    alpha, first = torch.rand((T, D), generator=g, device="cuda"), torch.randn((1, 1, D, V), generator=g, device="cuda")

    def run(columns, pieces=None):
        w = len(range(V)[columns])
        state, o = first[..., columns].clone(), torch.empty((T, w), device="cuda")
        k.linear_attention(o, torch.cat([qk, v[:, columns]], 1), 0, D, 2 * D, alpha, None, state, plan_of([T], [0]), 1, D, w, 0.3, pieces=pieces)
        return o, state
    o, state = run(slice(None))
    for columns in (slice(n), slice(V - n, None)):
        for a, b in zip((o[:, columns], state[..., columns]), run(columns, pieces=False)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("H,D,V,R", [(16, 32, 72, 40), (16, 20, 30, 40), (8, 64, 128, 16), (8, 48, 136, 16), (4, 128, 72, 16), (4, 100, 128, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("per_head", [False, True])
def test_a_batch_gives_the_bits_of_its_sequences_alone(H, D, V, R, dtype, per_head):
    """Many sequences of up to three tokens: a column a thread; each of them alone: four columns a thread.  The same sums in the same order."""
    from zlm_b200.kernels import get_kernels
    k = get_kernels()
    news = [1 + r % 3 for r in range(R)]
    T = sum(news)
    assert k.lib.zlm_linear_attention_by_columns(3, R, H, D, V) and not k.lib.zlm_linear_attention_by_columns(3, 1, H, D, V)
    g = torch.Generator(device="cuda").manual_seed(D + V)
    proj = torch.randn((T, 2 * H * D + H * V + 3), generator=g, device="cuda").to(dtype)
    alpha, head = torch.rand((T, H * D), generator=g, device="cuda"), torch.linspace(0.5, 0.99, H, device="cuda")
    first = torch.randn((R, H, D, V), generator=g, device="cuda")

    def run(rows, states, n):
        state, o = states.clone(), torch.full((rows.stop - rows.start, H * V), float("nan"), device="cuda")
        k.linear_attention(o, proj[rows], 0, H * D, 2 * H * D, None if per_head else alpha[rows], head if per_head else None, state,
                           plan_of(n, [5] * len(n)), H, D, V, 0.3)
        return o, state
    o, state = run(slice(0, T), first, news)
    assert not torch.isnan(o).any()
    at = 0
    for r, n in enumerate(news):
        slot = R - 1 - r                              # (plan_of hands the slots out in reverse)
        a, b = run(slice(at, at + n), first[slot:slot + 1], [n])
        assert torch.equal(a, o[at:at + n]) and torch.equal(b[0], state[slot])
        at += n
