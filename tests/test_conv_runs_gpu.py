"""Convolution, heads' norm and cache write in runs of tokens: bit for bit what the kernel of a token a warp gives (the same
step cut into chunks of fewer tokens than a run's rule wants, which is asked), over unequal sequences, carried inputs, padded heads, 2 to 5 taps."""
import pytest
import torch

from test_piece_products_gpu import plan_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv,dim,vdim,hdp", [(4, 2, 128, 128, 128), (3, 1, 48, 64, 64), (2, 2, 36, 20, 48)])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("norm", [True, False])
def test_runs_give_the_bits_of_single_tokens(nq, nkv, dim, vdim, hdp, taps, dtype, norm):
    from zlm_b200.kernels import PAGE_TOKENS, get_kernels
    k = get_kernels()
    g = torch.Generator(device="cuda").manual_seed(dim + taps)
    C = (nq + nkv) * dim + nkv * vdim
    news, starts = [1791, 1, 3, 131], [0, 70, 1, 64]
    proj = torch.randn((sum(news), C + 8), generator=g, device="cuda").to(dtype)
    w = torch.randn((C, taps), generator=g, device="cuda").to(dtype)
    R = len(news)
    pages = [-(-(n + s) // PAGE_TOKENS) for n, s in zip(news, starts)]
    table = torch.arange(R * max(pages), device="cuda", dtype=torch.int32).view(R, -1)
    first = torch.randn((R, taps - 1, C), generator=g, device="cuda").to(dtype)

    def run(chunks):
        """``chunks``: lists of new tokens by sequence, one list a step."""
        state, out = first.clone(), torch.full((sum(news), nq * hdp), float("nan"), device="cuda", dtype=dtype)
        pool = torch.zeros((table.numel(), 2, nkv, PAGE_TOKENS, hdp), device="cuda", dtype=dtype)
        done = [0] * R
        base = [sum(news[:r]) for r in range(R)]
        for step in chunks:
            live = [r for r in range(R) if step[r]]
            plan = plan_of([step[r] for r in live], [starts[r] + done[r] for r in live])
            slots = torch.tensor(live, device="cuda", dtype=torch.int32)
            plan.seq_slot, plan.token_slot = slots, slots[plan.token_seq.long()]
            rows = torch.cat([torch.arange(base[r] + done[r], base[r] + done[r] + step[r], device="cuda") for r in live])
            q = torch.full((len(rows), nq * hdp), float("nan"), device="cuda", dtype=dtype)
            k.conv_norm_write(q, proj[rows].contiguous(), w, state, plan, table, pool, nq, nkv, dim, vdim, taps, norm, 1e-6)
            out[rows] = q
            done = [d + n for d, n in zip(done, step)]
        assert done == news
        return out, state, pool
    whole = run([news])
    cut = [[min(97, max(0, n - 97 * i)) for n in news] for i in range(19)]
    units = nq + 2 * nkv
    assert k.lib.zlm_conv_runs(sum(news), R, units, hdp, taps)
    assert not any(k.lib.zlm_conv_runs(sum(step), sum(n > 0 for n in step), units, hdp, taps) for step in cut)
    for a, b in zip(whole, run(cut)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("off", [1, 2, 4])
def test_taps_that_start_off_a_read_of_four(taps, dtype, off):
    """Runs are taken wherever the taps start, and give the bits that they give of aligned taps."""
    from zlm_b200.kernels import PAGE_TOKENS, get_kernels
    k = get_kernels()
    nq, nkv, dim, vdim, T = 6, 2, 128, 64, 1031
    g = torch.Generator(device="cuda").manual_seed(taps)
    C = (nq + nkv) * dim + nkv * vdim
    proj = torch.randn((T, C), generator=g, device="cuda").to(dtype)
    taps_at = torch.zeros(C * taps + 16, device="cuda", dtype=dtype)
    values = torch.randn((C, taps), generator=g, device="cuda").to(dtype)
    first = torch.randn((1, taps - 1, C), generator=g, device="cuda").to(dtype)
    table = torch.arange(-(-T // PAGE_TOKENS), device="cuda", dtype=torch.int32).view(1, -1)
    assert k.lib.zlm_conv_runs(T, 1, nq + 2 * nkv, dim, taps)
    got = []
    for at in (0, off):
        w = taps_at[at:at + C * taps].view(C, taps)
        w.copy_(values)
        q, state = torch.empty((T, nq * dim), device="cuda", dtype=dtype), first.clone()
        pool = torch.zeros((table.numel(), 2, nkv, PAGE_TOKENS, dim), device="cuda", dtype=dtype)
        k.conv_norm_write(q, proj, w, state, plan_of([T], [0]), table, pool, nq, nkv, dim, vdim, taps, True, 1e-6)
        got.append((q, state, pool))
    for a, b in zip(*got):
        assert torch.equal(a, b)
