"""tcgen05 products on both sides of the lines where a whole warp issues them instead of a thread (12 or 24 stages of 64 columns
of K, 32 for tiles of 224 and 48 for wider ones; more than one token tile in blocks that stand alone), K off the stages' multiples, in every form: one round and persistent few-token blocks, pairs."""
import pytest
import torch

from zlm_b200.kernels import get_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N", [(40, 520), (300, 7000), (385, 1024), (600, 3584), (1000, 5130)])
@pytest.mark.parametrize("K", [64, 64 * 11, 64 * 11 + 8, 64 * 12, 64 * 24, 64 * 24 + 8, 64 * 47, 64 * 47 + 8, 64 * 48 + 40])
def test_products_around_the_lines(T, N, K):
    products(T, N, K)


@pytest.mark.parametrize("T,N", [(128, 3080), (129, 9000), (384, 6000), (384, 130), (700, 8192)])
@pytest.mark.parametrize("K", [64 * 11, 64 * 11 + 8, 64 * 23, 64 * 31, 64 * 31 + 8, 64 * 48 + 40])
def test_blocks_of_one_and_more_token_tiles(T, N, K):
    products(T, N, K)


def products(T, N, K):
    k = get_kernels()
    g = torch.Generator(device="cuda").manual_seed(T + K)
    x = torch.randn((T, K), generator=g, device="cuda").bfloat16()
    w = (torch.randn((N, K), generator=g, device="cuda") / K ** 0.5).bfloat16()
    first = torch.randn((T, N), generator=g, device="cuda")
    want = x.double() @ w.double().T
    got, acc = torch.empty((T, N), device="cuda"), first.clone()
    half = torch.empty((T, N), device="cuda", dtype=torch.bfloat16)
    k.linear(got, x, w)
    k.linear(acc, x, w, accumulate=True)
    k.linear(half, x, w)
    k.check_status(sync=True)
    # K products of the order of 1 / sqrt(K) summed in 32 bits; the bf16 result is rounded once more (2^-9 of it)
    assert (got.double() - want).abs().max() < 4e-5
    assert (acc.double() - first.double() - want).abs().max() < 4e-5
    assert ((half.double() - want).abs() <= want.abs() * 2.0 ** -8 + 4e-5).all()
