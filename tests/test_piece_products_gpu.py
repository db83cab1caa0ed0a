"""Recurrences over pieces of a prompt as tensor-core products of fp32 numbers cut into bfloat16 pieces, beside 64-bit walks
of the same inputs: lengths around a piece's edges, heads narrower and wider than a tile, partial rotations, states carried in.

Bounds.  The results are sums of some hundred fp32 products whose roundings are independent: 2^-24 of each, a few 1e-7 of the
result's norm; 1e-6 leaves a factor of four.  Gated outputs are rounded to bfloat16 (2^-9 of each number, at most): 4e-3."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def plan_of(news, starts):
    from zlm_b200.parts.base import Workspace
    ws, R = Workspace("cuda"), len(news)

    def ints(v):
        return torch.as_tensor(v, dtype=torch.int32, device="cuda")
    pos = torch.cat([torch.arange(s, s + n) for n, s in zip(news, starts)])
    seq = torch.cat([torch.full((n,), r) for r, n in enumerate(news)])
    return types.SimpleNamespace(
        R=R, T=sum(news), cu_seqlens=ints([0] + torch.tensor(news).cumsum(0).tolist()), seq_slot=ints(list(range(R))[::-1]),
        seq_start=ints(starts), seq_new=ints(news), token_pos=ints(pos), token_slot=ints(R - 1 - seq), token_seq=ints(seq),
        max_new=max(news), max_len=max(n + s for n, s in zip(news, starts)), is_decode=False, scratch=ws.get)


def close(got, want, rel):
    assert torch.isfinite(got).all()
    assert (got.double() - want).norm() <= rel * want.norm(), f"{((got.double() - want).norm() / want.norm()).item():.2e}"


def calls(k, monkeypatch):
    """The names of the library's entry points, as ``k`` calls them from here on."""
    names, call = [], k._call

    def noted(name, *args):
        names.append(name)
        return call(name, *args)
    monkeypatch.setattr(k, "_call", noted)
    return names


def unit(o):
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)


@pytest.mark.parametrize("H,D,V,n_rot", [(2, 128, 128, 128), (3, 64, 72, 32), (1, 16, 8, 0), (2, 96, 136, 96), (1, 112, 64, 16)])
@pytest.mark.parametrize("news,starts", [([256], [0]), ([257, 1, 64], [0, 5, 300]), ([63, 321], [9, 0])])
@pytest.mark.parametrize("table", [True, False])
def test_retention(H, D, V, n_rot, news, starts, table, monkeypatch):
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
    assert k.lib.zlm_retention_products(1, 2 * H * (D + V), 0, H * D, 2 * H * D, n_rot, D, V)
    T = plan.T
    g = torch.Generator(device="cuda").manual_seed(D + V + T)
    proj = torch.randn((T, 2 * H * D + 2 * H * V), generator=g, device="cuda").bfloat16()
    decay = torch.linspace(0.9, 0.999, H, device="cuda")
    inv = torch.pow(1e4, -torch.arange(n_rot // 2, device="cuda").double() / max(1, n_rot // 2)).float()
    first = torch.randn((plan.R, H, D, V), generator=g, device="cuda")
    cos_sin = None
    if table and n_rot:
        cos_sin = torch.empty((2, n_rot // 2, T), device="cuda")
        k.rope_table(cos_sin, inv, n_rot, plan.token_pos)
    # (angles as the kernels form them, in fp32: what they are off at large positions is not this test's matter)
    a = (plan.token_pos[:, None].float() * inv).double()[:, None]

    def turn(x):
        u, v = x[..., :n_rot // 2], x[..., n_rot // 2:n_rot]
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., n_rot:]], -1)
    q, key = (turn(proj[:, i * H * D:(i + 1) * H * D].double().view(T, H, D)) for i in (0, 1))
    key = key * D ** -0.5
    v = proj[:, 2 * H * D:2 * H * D + H * V].double().view(T, H, V)
    want, S = torch.empty((T, H, V), dtype=torch.float64, device="cuda"), first.double()
    at = 0
    for r, n in enumerate(news):
        s = S[plan.R - 1 - r]
        for t in range(at, at + n):
            s = decay.double()[:, None, None] * s + key[t][:, :, None] * v[t][:, None]
            want[t] = (s * q[t][:, :, None]).sum(1)
        S[plan.R - 1 - r] = s
        at += n
    gate = proj[:, 2 * H * D + H * V:]
    args = (proj, 0, H * D, 2 * H * D, inv if n_rot else None, n_rot, decay)
    state, o = first.clone(), torch.full((T, H * V), float("nan"), device="cuda")
    k.retention(o, *args, state, plan, H, D, V, D ** -0.5, cos_sin=cos_sin)
    close(o, want.flatten(1), 1e-6)
    close(state, S, 1e-6)
    state, y = first.clone(), torch.full((T, H * V), float("nan"), device="cuda", dtype=torch.bfloat16)
    names = calls(k, monkeypatch)
    k.retention_gated(y, gate, 1e-6, "silu", o, *args, state, plan, H, D, V, D ** -0.5, cos_sin=cos_sin)
    assert names == ["zlm_retention_parts"] + ["zlm_head_gate"] * (V > 128)        # (a head wider than a block norms elsewhere)
    z = gate.double()
    close(y, unit(want).flatten(1) * z * torch.sigmoid(z), 4e-3)
    close(state, S, 1e-6)


@pytest.mark.parametrize("H,D,V,cap", [(2, 128, 128, 15.0), (3, 64, 72, 0.0), (1, 16, 8, 15.0), (2, 96, 136, 15.0)])
@pytest.mark.parametrize("news,starts", [([64], [0]), ([65, 1, 130], [0, 5, 300]), ([17, 2], [9, 0])])
@pytest.mark.parametrize("spread", [1.0, 8.0])
def test_matrix_memory(H, D, V, cap, news, starts, spread, monkeypatch):
    """``spread``: the gates' logits times that: forget gates near 0 and 1, running maxima that jump.  Outputs are quotients
    whose denominator is a sum of either sign: one that is a hundredth of its terms carries their roundings a hundredfold, and a
    few of a head's 19 to 200 rows are like that (4e-6 over all rows; with gates spread wide one token decides a row: 1e-4)."""
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
    T = plan.T
    gen = torch.Generator(device="cuda").manual_seed(D + V + T)
    assert k.lib.zlm_mlstm_products(1, 2 * H * (D + V), 0, H * D, 2 * H * D, D, V)
    names = calls(k, monkeypatch)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda")
    proj, z = rand(T, 2 * H * D + 2 * H * V).bfloat16(), rand(T, 2 * H) * spread
    b_i, b_f = rand(H), rand(H) + 2
    first = (rand(plan.R, H, D, V) * 0.3, rand(plan.R, H, D), rand(plan.R, H).abs())
    q, key = (proj[:, i * H * D:(i + 1) * H * D].double().view(T, H, D) for i in (0, 1))
    q = q * D ** -0.5
    v = proj[:, 2 * H * D:2 * H * D + H * V].double().view(T, H, V)

    def capped(x):
        return cap * torch.tanh(x / cap) if cap else x
    gi = capped(z[:, :H].double() + b_i.double())
    gf = torch.nn.functional.logsigmoid(capped(z[:, H:].double() + b_f.double()))
    want = torch.empty((T, H, V), dtype=torch.float64, device="cuda")
    S, N, M = (t.double() for t in first)
    at = 0
    for r, n in enumerate(news):
        s, nv, m = (t[plan.R - 1 - r] for t in (S, N, M))
        for t in range(at, at + n):
            new = torch.maximum(gf[t] + m, gi[t])
            a, b = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new)
            s = a[:, None, None] * s + b[:, None, None] * key[t][:, :, None] * v[t][:, None]
            nv, m = a[:, None] * nv + b[:, None] * key[t], new
            want[t] = (s * q[t][:, :, None]).sum(1) / (torch.maximum((nv * q[t]).sum(1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        S[plan.R - 1 - r], N[plan.R - 1 - r], M[plan.R - 1 - r] = s, nv, m
        at += n
    gate = proj[:, 2 * H * D + H * V:]
    for gated in (False, True):
        state = tuple(t.clone() for t in first)
        args = (proj, 0, H * D, 2 * H * D, z, 0, H, b_i, b_f, cap, state, plan, H, D, V, D ** -0.5)
        o = torch.full((T, H * V), float("nan"), device="cuda")
        if gated:
            y = torch.full((T, H * V), float("nan"), device="cuda", dtype=torch.bfloat16)
            w = torch.rand((H * V,), generator=gen, device="cuda") + 0.5
            names.clear()
            k.mlstm_gated(y, gate, w, 1e-6, o, *args)
            assert names == ["zlm_mlstm"] + ["zlm_norm_gate"] * (V > 128)
            close(y, unit(want).flatten(1) * w.double() * torch.sigmoid(gate.double()), 4e-3)
        else:
            k.mlstm(o, *args)
            close(o, want.flatten(1), 4e-6 if spread == 1.0 else 1e-4)
        for got, exact in zip(state, (S, N, M)):
            close(got, exact, 1e-6)


def kinds(x):
    """0 where finite, 1 / -1 for infinities, 2 for NaN."""
    x = x.double()
    return torch.where(torch.isnan(x), 2.0, torch.where(torch.isinf(x), torch.sign(x), 0.0))


# where a number that is not finite stands: the operand's columns of the projection (or the state), the token, the column
@pytest.mark.parametrize("where", ["query", "key", "value", "state"])
@pytest.mark.parametrize("number", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("token", [0, 8, 21, 63, 70, 255])
@pytest.mark.parametrize("part", ["retention", "matrix memory"])
def test_numbers_that_are_not_finite_reach_what_sees_them(part, where, number, token):
    """Tokens ahead of such a number, and columns that it does not enter, keep their results to the bit; what it enters is not
    finite, and behind a key or a state it is the infinity or NaN of a 64-bit walk over the tokens (behind a query or a value that
    depends on the order of the sums: infinities of both signs meet where a state is read, or do not where scores are)."""
    from zlm_b200.kernels import get_kernels
    k, H, D, V, T = get_kernels(), 2, 64, 72, 256
    plan = plan_of([T], [0])
    g = torch.Generator(device="cuda").manual_seed(5)

    def rand(*shape):
        return torch.randn(shape, generator=g, device="cuda")
    clean = (rand(T, 2 * H * D + 2 * H * V)).bfloat16()
    # (forget gates near one: a weight that underflows times an infinity is NaN in any order of the sums)
    z = torch.cat([rand(T, H), rand(T, H) + 7], 1)
    first = [rand(1, H, D, V) * 0.3, rand(1, H, D), rand(1, H).abs()]
    decay = torch.linspace(0.9, 0.99, H, device="cuda")
    col = {"query": 5, "key": H * D + 5, "value": 2 * H * D + 5, "state": 0}[where]
    spoilt, spoilt_first = clean.clone(), first[0].clone()
    if where == "state":
        spoilt_first[0, 0, 7, 5] = number
    else:
        spoilt[token, col] = number                  # (head 0)

    def run(proj, S, gated):
        state = [S.clone(), first[1].clone(), first[2].clone()]
        o = torch.zeros((T, H * V), device="cuda")
        y = torch.zeros((T, H * V), device="cuda", dtype=torch.bfloat16)
        gate = proj[:, 2 * H * D + H * V:]
        if part == "retention":
            args = (o, proj, 0, H * D, 2 * H * D, None, 0, decay, state[0], plan, H, D, V, 0.125)
            k.retention_gated(y, gate, 1e-6, "silu", *args) if gated else k.retention(*args)
        else:
            args = (o, proj, 0, H * D, 2 * H * D, z, 0, H, None, None, 15.0, state, plan, H, D, V, 0.125)
            w = torch.ones((H * V,), device="cuda")
            k.mlstm_gated(y, gate, w, 1e-6, *args) if gated else k.mlstm(*args)
        return (y if gated else o).view(T, H, V), state[0]

    def walk(proj, S0):
        q, key = (proj[:, i * H * D:(i + 1) * H * D].double().view(T, H, D) for i in (0, 1))
        v = proj[:, 2 * H * D:2 * H * D + H * V].double().view(T, H, V)
        S, out = S0[0].double(), []
        n, m = first[1][0].double(), first[2][0].double()
        gi, gf = 15 * torch.tanh(z[:, :H].double() / 15), torch.nn.functional.logsigmoid(15 * torch.tanh(z[:, H:].double() / 15))
        for t in range(T):
            if part == "retention":
                a, b, den = decay.double(), torch.full((H,), 0.125, dtype=torch.float64, device="cuda"), torch.ones(H, 1, device="cuda")
            else:
                new = torch.maximum(gf[t] + m, gi[t])
                a, b, m = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new), new
                n = a[:, None] * n + b[:, None] * key[t]
                den = torch.maximum((n * q[t] * 0.125).sum(1).abs(), torch.exp(-m))[:, None] + 1e-6
            S = a[:, None, None] * S + b[:, None, None] * key[t][:, :, None] * v[t][:, None]
            out.append((S * q[t][:, :, None] * (1.0 if part == "retention" else 0.125)).sum(1) / den)
        return torch.stack(out), S[None]
    sees = torch.zeros((T, H, V), dtype=torch.bool, device="cuda")       # outputs that the number enters
    if where == "query":
        sees[token, 0] = True
    elif where == "key":
        sees[token:, 0] = True
    elif where == "value":
        sees[token:, 0, 5] = True
    else:
        sees[:, 0, 5] = True
    (o, S), (o_clean, S_clean) = run(spoilt, spoilt_first, False), run(clean, first[0], False)
    want, S_want = walk(spoilt, spoilt_first)
    assert torch.equal(o[~sees], o_clean[~sees])
    if where in ("key", "state"):
        assert torch.equal(kinds(o), kinds(want))
    assert not torch.isfinite(o[sees]).any() and not torch.isfinite(want[sees]).any()
    assert torch.equal(kinds(S), kinds(S_want))
    fine = kinds(S_want) == 0
    assert torch.equal(S[fine], S_clean[fine])
    y, _ = run(spoilt, spoilt_first, True)
    y_clean, _ = run(clean, first[0], True)
    rows = ~sees.any(2)                                                   # (a head's norm takes all its columns along)
    assert torch.equal(y[rows], y_clean[rows])
    assert (kinds(y[~rows]) != 0).any(1).all()
