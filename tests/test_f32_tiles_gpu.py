"""32-bit attention in tiles of 32 queries: bit for bit what the kernel of one block a query gives, over lengths around a
tile's and a chunk's edges, cached beginnings, windows, chunks of positions and sinks."""
import types

import pytest
import torch

from test_piece_products_gpu import calls

pytestmark = pytest.mark.gpu


def _case(nq, nkv, hd, news, starts, seed=0):
    from zlm_b200.kernels import PAGE_TOKENS
    g = torch.Generator(device="cuda").manual_seed(seed)
    need = [-(-(n + s) // PAGE_TOKENS) for n, s in zip(news, starts)]
    table = torch.zeros((len(news), max(need)), dtype=torch.int32)
    order = torch.randperm(sum(need) + 1, generator=torch.Generator().manual_seed(seed)).tolist()
    at = 0
    for r, n in enumerate(need):
        table[r, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    # what no token wrote is not a number: nothing of it may reach a result
    pool = torch.full((sum(need) + 1, 2, nkv, PAGE_TOKENS, hd), float("nan"), device="cuda")
    for r, (n, s) in enumerate(zip(news, starts)):
        t = torch.arange(n + s, device="cuda")
        pages = table[r].cuda().long()[t // PAGE_TOKENS]
        for j in (0, 1):
            pool[pages, j, :, t % PAGE_TOKENS] = torch.randn((n + s, nkv, hd), generator=g, device="cuda")
    cu = torch.tensor([0] + list(torch.tensor(news).cumsum(0)), dtype=torch.int32, device="cuda")
    pos = torch.cat([torch.arange(s, s + n) for n, s in zip(news, starts)]).int().cuda()
    slot = torch.cat([torch.full((n,), r) for r, n in enumerate(news)]).int().cuda()
    T = sum(news)
    qkv = torch.randn((T, (nq + 2) * hd), generator=g, device="cuda")
    plan = types.SimpleNamespace(is_decode=False, cu_seqlens=cu, seq_slot=torch.arange(len(news), device="cuda").int(),
                                 seq_start=torch.tensor(starts, dtype=torch.int32, device="cuda"), R=len(news), max_new=max(news),
                                 max_len=max(1 << 20, max(news)))       # (long enough for tiles whatever the sizes are)
    return qkv[:, :nq * hd], pool, table.cuda(), pos, slot, plan


@pytest.mark.parametrize("nq,nkv,hd", [(4, 2, 128), (3, 1, 64), (2, 2, 96)])
@pytest.mark.parametrize("news,starts", [([8], [0]), ([31, 1, 33], [0, 200, 31]), ([129], [515]), ([40, 64], [1, 64]), ([1, 1], [700, 3])])
@pytest.mark.parametrize("window,chunk,sink", [(0, 0, None), (40, 0, True), (1, 0, "numbers"), (0, 48, None), (100, 0, None)])
def test_tiles_give_the_bits_of_single_queries(nq, nkv, hd, news, starts, window, chunk, sink, monkeypatch):
    from zlm_b200.kernels import get_kernels
    k = get_kernels()
    q, pool, table, pos, slot, plan = _case(nq, nkv, hd, news, starts)
    sinks = torch.linspace(-2, 2, nq, device="cuda") if sink == "numbers" else None
    outs, names = [], calls(k, monkeypatch)
    for p in (None, plan):
        out = torch.full((q.shape[0], nq * hd), float("nan"), device="cuda")
        k.attention(out, q, pool, table, pos, slot, nq, nkv, hd, hd ** -0.5, window, p, sink=bool(sink), sinks=sinks, chunk=chunk)
        outs.append(out)
    assert names == ["zlm_attention_generic", "zlm_attention_f32_tile"]
    assert not torch.isnan(outs[0]).any()
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))


@pytest.mark.parametrize("T,N,K", [(1, 1, 1), (63, 65, 31), (65, 64, 33), (130, 70, 66), (64, 128, 256), (3, 200, 2048)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_product_at_the_edges_of_its_tiles(T, N, K, accumulate):
    """A 32-bit sum of K products of order one is off by at most K roundings of a partial sum of order sqrt(K): 2^-24 K."""
    from zlm_b200.kernels import get_kernels
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    x, w = torch.randn((T, K), generator=g, device="cuda"), torch.randn((N, K), generator=g, device="cuda")
    y = torch.randn((T, N), generator=g, device="cuda")
    want = x.double() @ w.double().T + (y.double() if accumulate else 0)
    bits = y.clone()
    get_kernels().linear(y, x, w, accumulate=accumulate)
    assert ((y.double() - want).abs() <= 2.0 ** -24 * (K + 4) * max(1.0, K ** 0.5) * 2).all()
    # a token's result does not depend on the tokens beside it
    get_kernels().linear(bits[T // 2:T // 2 + 1], x[T // 2:T // 2 + 1], w, accumulate=accumulate)
    assert torch.equal(bits[T // 2], y[T // 2])


@pytest.mark.parametrize("T,N,K", [(1, 64, 32), (65, 130, 100), (64, 64, 2048)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_products_of_operands_off_their_alignment_are_the_same_bits(T, N, K, accumulate):
    """An operand that starts 4 bytes late takes the kernel of single columns: the same sums in the same order."""
    from zlm_b200.kernels import get_kernels
    k = get_kernels()
    g = torch.Generator(device="cuda").manual_seed(T)
    x, w = torch.randn((T, K), generator=g, device="cuda"), torch.randn((N, K), generator=g, device="cuda")
    y = torch.randn((T, N), generator=g, device="cuda")
    want = y.clone()
    k.linear(want, x, w, accumulate=accumulate)
    for late in ("x", "w"):
        a, b = (torch.empty(t.numel() + 1, device="cuda")[1:].view_as(t).copy_(t) if n == late else t for n, t in (("x", x), ("w", w)))
        assert (a.data_ptr() | b.data_ptr()) % 16 == 4
        got = y.clone()
        k.linear(got, a, b, accumulate=accumulate)
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
