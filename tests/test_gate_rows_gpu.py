"""Heads times a gate without a norm: rows of neighbouring heads take eight numbers a thread and give the bits of the form of a
warp a head (which heads with padding between them take), at rows of few and many numbers, logits at both ends among them."""
import pytest
import torch

from zlm_b200.kernels import get_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", ["sigmoid", "silu"])
@pytest.mark.parametrize("T,H,V", [(1, 1, 8), (3, 3, 24), (257, 5, 128), (2999, 16, 128), (33, 2, 512)])
@pytest.mark.parametrize("in_place", [False, True])
def test_rows_equal_heads(T, H, V, act, in_place):
    k = get_kernels()
    g = torch.Generator(device="cuda").manual_seed(T + V)
    o = torch.randn((T, H, V), generator=g, device="cuda").bfloat16()
    wide = torch.randn((T, H * V + 16), generator=g, device="cuda").mul(4).bfloat16()
    wide[0, :8] = torch.tensor([float("inf"), -float("inf"), 3e38, -3e38, 90.0, -90.0, 0.0, -0.0])
    gate = wide[:, :H * V]
    padded = torch.zeros((T, H, V + 8), device="cuda", dtype=torch.bfloat16)
    padded[:, :, :V] = o
    want = torch.empty((T, H * V), device="cuda", dtype=torch.bfloat16)
    k.head_gate(want, padded[:, :, :V], gate, H, V, False, 0.0, act)
    got = o.view(T, H * V) if in_place else torch.empty_like(want)
    k.head_gate(got, o, gate, H, V, False, 0.0, act)
    same = (got == want) | (torch.isnan(got) & torch.isnan(want))
    assert same.all()
    z = gate[1:].double() if T > 1 else gate[:, 8:].double()
    v = padded[:, :, :V].reshape(T, -1).double()
    v = v[1:] if T > 1 else v[:, 8:]
    ref = v * torch.sigmoid(z) * (z if act == "silu" else 1.0)
    mine = (got[1:] if T > 1 else got[:, 8:]).double()
    assert ((mine - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-30).all()         # one rounding to bfloat16, and 32-bit functions


@pytest.mark.parametrize("off,pad", [(0, 4), (4, 0), (1, 0), (8, 8), (0, 1)])
@pytest.mark.parametrize("which", ["out", "o", "g"])
def test_rows_off_sixteen_bytes(off, pad, which):
    """Starts and strides that are no multiple of eight numbers go to the form of a warp a head, with the same bits."""
    k = get_kernels()
    T, H, V = 65, 4, 128
    N = H * V
    g = torch.Generator(device="cuda").manual_seed(off + pad)
    values = {n: torch.randn((T, N), generator=g, device="cuda").bfloat16() for n in ("out", "o", "g")}

    def placed(name):
        if name != which:
            return values[name].clone()
        t = torch.zeros(T * (N + pad) + off, device="cuda", dtype=torch.bfloat16)[off:].as_strided((T, N), (N + pad, 1))
        return t.copy_(values[name])

    want = torch.empty((T, N), device="cuda", dtype=torch.bfloat16)
    k.head_gate(want, values["o"].view(T, H, V), values["g"], H, V, False, 0.0, "silu")
    out, o, gate = placed("out"), placed("o"), placed("g")
    k.head_gate(out, o.as_strided((T, H, V), (o.stride(0), V, 1)), gate, H, V, False, 0.0, "silu")
    assert torch.equal(out, want)
