"""The routed experts' sorted products at the edges of their tiles (256 rows of W, up to 256 sorted rows, 32 columns an
epilogue turn, 64 of K), and products of few outputs over many tokens, which are cut along K."""
import pytest
import torch

from zlm_b200.kernels import get_kernels, interleave_gate_up

pytestmark = pytest.mark.gpu


def routed(counts, identities, top, seed):
    """idx [T, top] in which expert e stands counts[e] times and an index beyond the experts ``identities`` times."""
    g = torch.Generator().manual_seed(seed)
    flat = torch.cat([torch.full((n,), e) for e, n in enumerate(counts + [identities])])
    assert len(flat) % top == 0
    return flat[torch.randperm(len(flat), generator=g)].view(-1, top).to(torch.int32)


# (rows of every expert, identities, choices a token, hidden size, channels of an expert)
CASES = [
    ([1, 0, 31, 32, 33, 0, 64, 7], 0, 2, 64, 32),
    ([255, 256, 257, 0, 1, 512, 513, 300], 12, 3, 72, 136),          # tails of W's tiles and of K
    ([0, 0, 0, 40], 0, 4, 128, 128),
    ([2, 3, 5, 1030, 8], 6, 17, 264, 264),                           # more choices a token than a thread keeps places for
    ([1] * 40, 0, 1, 256, 64),
]


@pytest.mark.parametrize("activation", ["relu2", "swiglu_interleaved", "swish_limit_interleaved"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_sorted_experts_against_64_bits(case, activation):
    counts, identities, top, W, F = CASES[case]
    k, E = get_kernels(), len(counts)
    idx = routed(counts, identities, top, case)
    T = idx.shape[0]
    g = torch.Generator().manual_seed(100 + case)
    rnd = lambda *s: torch.randn(*s, generator=g)
    x, wgt = rnd(T, W).bfloat16(), torch.rand(T, top, generator=g) + 0.1
    gate, up, down = (rnd(E, F, W) / W ** 0.5).bfloat16(), (rnd(E, F, W) / W ** 0.5).bfloat16(), (rnd(E, W, F) / F ** 0.5).bfloat16()
    start = rnd(T, W)
    gated = activation != "relu2"
    w_up = torch.stack([interleave_gate_up(a, b) for a, b in zip(gate, up)]) if gated else up
    got = start.clone().cuda()
    k.moe_grouped(got, x.cuda(), w_up.cuda(), down.cuda(), idx.cuda(), wgt.cuda(), scale_input=not gated, impl="tc",
                  activation=activation, identity=True, limit=2.0, alpha=1.5)
    k.check_status(sync=True)
    want = start.double()
    bf = lambda t: t.to(torch.bfloat16).double()                     # what the two products hand on is rounded once each
    for t in range(T):
        for e, w in zip(idx[t].tolist(), wgt[t].double()):
            h = x[t].double()
            if e >= E:
                want[t] += w * h
                continue
            if not gated:
                a = torch.relu(up[e].double() @ bf((h * w).float())) ** 2
            else:
                z, v = gate[e].double() @ h, up[e].double() @ h
                if activation == "swiglu_interleaved":
                    a = z * torch.sigmoid(z) * v
                else:
                    z, v = z.clamp(max=2.0), v.clamp(-2.0, 2.0)
                    a = z * torch.sigmoid(1.5 * z) * (v + 1)
            want[t] += (down[e].double() @ bf(a.float())) * (w if gated else 1.0)
    # fp32 sums may move an activation to the neighbouring bf16 value (2^-8 of it, few of them); a row of another expert, a
    # missing choice or a column out of place would be of the order of the row itself
    rel = ((got.cpu().double() - want).norm(dim=1) / want.norm(dim=1)).max()
    assert rel < 2e-3, f"case {case} {activation}: a token is {rel:.2e} off"


@pytest.mark.parametrize("T, N, K", [(385, 8, 512), (2048, 64, 2048), (2047, 33, 1032), (4097, 128, 1024), (9472, 16, 1024), (9473, 16, 1024)])
def test_few_outputs_over_many_tokens(T, N, K):
    k = get_kernels()
    assert (k.lib.zlm_gemm_tc_ksplit(T, N, K) > 1) == (T <= 9472 and K >= 1024)
    g = torch.Generator().manual_seed(T + N)
    x, w = torch.randn(T, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    first = torch.randn(T, N, generator=g)
    got, acc = torch.empty(T, N, device="cuda"), first.cuda()
    k.linear(got, x.cuda(), w.cuda())
    k.linear(acc, x.cuda(), w.cuda(), accumulate=True)
    k.flush_shares()
    k.check_status(sync=True)
    # sums of K products of the order of 1 / sqrt(K) in 32 bits
    assert (got.cpu().double() - want).abs().max() < 2e-5
    assert (acc.cpu().double() - first.double() - want).abs().max() < 2e-5


@pytest.mark.parametrize("T, N, K", [(385, 8, 1024), (1500, 64, 1536), (1024, 64, 1544), (3000, 128, 2048), (4097, 32, 2048), (9472, 16, 1024)])
def test_few_outputs_over_many_tokens_in_bfloat16(T, N, K):
    """Cut along K or whole, by what is faster: both sides of that line."""
    k = get_kernels()
    g = torch.Generator().manual_seed(T + N)
    x, w = torch.randn(T, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    got = torch.empty(T, N, device="cuda", dtype=torch.bfloat16)
    k.linear(got, x.cuda(), w.cuda())
    k.check_status(sync=True)
    # one rounding to bf16 (2^-9 of the value) of sums in 32 bits
    assert ((got.cpu().double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-5).all()
