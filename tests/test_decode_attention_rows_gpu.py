"""Decode attention around the edges of a page: what is read before the wait for the kernel before (pages without a row of the
step's own, and the older rows of a sequence of one page) and after it give the bits of reading everything after it, whatever
the group, the head size and the split."""
import pytest
import torch

from zlm_b200.kernels import PAGE_TOKENS, get_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv,hd", [(2, 2, 16), (4, 2, 128), (10, 2, 96), (16, 1, 128), (9, 1, 64)])
@pytest.mark.parametrize("splits,per", [(1, 8), (8, 1), (3, 2)])
def test_rows_read_early_and_late(nq, nkv, hd, splits, per):
    from ctypes import c_float
    k = get_kernels()
    ends = [0, 1, 62, 63, 64, 65, 126, 127, 128, 129, 300, 383]
    if splits * per < 6:
        ends = [e for e in ends if e // PAGE_TOKENS < splits * per]
    T = len(ends)
    g = torch.Generator(device="cuda").manual_seed(nq * hd)
    pages = 6
    pool = torch.randn((T * pages, 2, nkv, PAGE_TOKENS, hd), generator=g, device="cuda").bfloat16()
    table = torch.randperm(T * pages, generator=g, device="cuda").int().view(T, pages).contiguous()
    pos = torch.tensor(ends, dtype=torch.int32, device="cuda")
    slot = torch.arange(T, dtype=torch.int32, device="cuda")
    q = torch.randn((T, nq * hd), generator=g, device="cuda").bfloat16()
    newest = torch.randn((T, 2, nkv, hd), generator=g, device="cuda").bfloat16()
    for t, e in enumerate(ends):                       # (in the place of what the kernel before is about to write)
        pool[table[t, e // PAGE_TOKENS].long(), :, :, e % PAGE_TOKENS] = 1000.0
    stale, got = pool.clone(), []
    part_o, part_ml = torch.empty(T * nq * splits * hd, device="cuda"), torch.empty(T * nq * splits * 2, device="cuda")

    def write(dst):
        # one kernel of the library that writes the newest rows: dependent launches put the attention's first reads beside it
        qkv = torch.cat([q, newest[:, 0].reshape(T, -1), newest[:, 1].reshape(T, -1)], 1).contiguous()
        k.qk_norm_rope_write(qkv, None, None, 0.0, None, 0, pos, slot, table, dst, nq, nkv, hd)

    for fresh in (0, 1, 70):
        pool.copy_(stale)
        out = torch.full((T, nq * hd), float("nan"), device="cuda").bfloat16()
        torch.cuda.synchronize()
        k.set_pdl(True)
        try:
            write(pool)
            k._call("zlm_attention_decode_fresh", k._at(out), out.stride(0), k._at(q), q.stride(0), k._at(pool), k._at(table), pages,
                    k._at(pos), k._at(slot), T, nq, nkv, hd, c_float(hd ** -0.5), 0, splits, per, k._at(part_o), k._at(part_ml), fresh,
                    0, 0, c_float(0.0), None, 1, 0, None, 0, k._queue())
        finally:
            k.set_pdl(False)
        got.append(out)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    for t, e in enumerate(ends):
        rows = torch.arange(e + 1, device="cuda")
        kv = pool[table[t].long()[rows // PAGE_TOKENS], :, :, rows % PAGE_TOKENS].double()           # [n, 2, nkv, hd]
        qq = q[t].double().view(nkv, nq // nkv, hd)
        p = torch.softmax(torch.einsum("ghd,ngd->ghn", qq, kv[:, 0]) * hd ** -0.5, -1)
        want = torch.einsum("ghn,ngd->ghd", p, kv[:, 1]).reshape(-1)
        # bfloat16 weights of the values and a bfloat16 result: 2^-8 of the row's size each, as one distance
        assert (got[1][t].double() - want).norm() < 2 ** -7 * want.norm(), f"position {e}"
