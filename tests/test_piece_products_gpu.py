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


def unit(o):
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)


@pytest.mark.parametrize("H,D,V,n_rot", [(2, 128, 128, 128), (3, 64, 72, 32), (1, 16, 8, 0), (2, 96, 136, 96), (1, 112, 64, 16)])
@pytest.mark.parametrize("news,starts", [([256], [0]), ([257, 1, 64], [0, 5, 300]), ([63, 321], [9, 0])])
@pytest.mark.parametrize("table", [True, False])
def test_retention(H, D, V, n_rot, news, starts, table):
    from zlm_b200.kernels import get_kernels
    k, plan = get_kernels(), plan_of(news, starts)
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
    k.retention_gated(y, gate, 1e-6, "silu", o, *args, state, plan, H, D, V, D ** -0.5, cos_sin=cos_sin)
    z = gate.double()
    close(y, unit(want).flatten(1) * z * torch.sigmoid(z), 4e-3)
    close(state, S, 1e-6)
