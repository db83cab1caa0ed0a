"""The host-side choices of the kernel library that need no GPU: how the weight-streaming
product spreads K over its warps and how many warps its blocks have, and into how many shares of K the few-token tcgen05
product cuts the tiles that do not fill a round of the GPU.  The library loads without a
GPU (it is compiled at the first call, a few seconds, if this checkout has not built it
yet); without nvcc the tests are skipped."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from zlm_b200.csrc.build import find_nvcc, library_path
    try:
        find_nvcc()
    except Exception as e:                          # no compiler here: nothing to test against
        pytest.skip(f"nvcc is not available: {e}")
    return ctypes.CDLL(library_path(build_if_needed=True, verbose=False))


@pytest.mark.parametrize("K,seg", [(4096, 512), (8192, 512), (12288, 512),          # multiples of 4096: 512, the order
                                   (1024, 128), (2048, 256), (3072, 384),            # the persistent kernel adds in
                                   (5120, 640), (25600, 640), (6144, 384), (7168, 128),
                                   (1000, 512), (520, 512), (4104, 512), (64, 512)])  # ragged: 512 and a tail
def test_gemv_segment_spreads_k_evenly(lib, K, seg):
    assert lib.zlm_gemv_segment(K) == seg
    if K % 1024 == 0:
        assert K % (8 * seg) == 0                   # whole chunks of 8 warps x seg columns: no warp idles


@pytest.mark.parametrize("N,K,narrow,warps", [
    (4096, 4096, 5, 8), (4096, 12288, 5, 8), (3072, 1024, 5, 8),   # one round of wide blocks: wide
    (6144, 4096, 5, 4),          # 384 blocks: the 88 after the first round of 296 would run alone
    (10240, 5120, 5, 4), (5120, 8192, 5, 4), (6144, 1024, 5, 4),
    (12800, 4096, 5, 8),         # 800 blocks: 740 narrow ones at once would leave 60 with half the loads in flight
    (24576, 4096, 5, 8),         # 1,536: five rounds of wide blocks and a short one, or two of narrow and a short one
    (24576, 4096, 4, 4),         # with two token tiles four narrow blocks fit: 592 + 592 + 352
    (10240, 5120, 4, 8),
])
def test_gemv_block_width_by_the_estimate_of_both_forms(lib, N, K, narrow, warps):
    """Each case was timed on a B200 in both forms; the estimate names the faster one (or either,
    where they were within a twentieth)."""
    assert lib.zlm_gemv_plan_warps(N, K, 148, 2, narrow) == warps
    assert lib.zlm_gemv_plan_warps(N, K, 0, 2, narrow) == 8        # nothing known about the device: wide


@pytest.mark.parametrize("T,N,K,shares", [
    (64, 6144, 4096, 3),        # 48 tiles: three shares fill 144 of 148 SMs
    (64, 4096, 4096, 4),        # 32 tiles x 4
    (64, 4096, 12288, 4),
    (64, 24576, 4096, 3),       # 192 tiles: 148 in one piece, 44 x 3 shares
    (64, 151936, 4096, 8),      # 1,187 tiles: 8 rounds in one piece, the last 3 tiles x 8
    (64, 18944, 4096, 1),       # 148 tiles: exactly one round, nothing to cut
    (300, 8000, 1024, 2),       # three token tiles per output tile; shares of at least 8 k blocks
    (40, 4096, 264, 1),         # K too short to cut
    (2048, 4096, 4096, 1),      # many tokens: the persistent forms, no shares
])
def test_few_token_shares_of_k(lib, T, N, K, shares):
    assert lib.zlm_gemm_tc_ksplit(T, N, K) == shares


@pytest.mark.parametrize("T,K,shares,bf16", [
    (384, 1024, 2, 1), (385, 1024, 2, 0), (9472, 1024, 2, 0), (385, 512, 1, 0),      # up to 384 tokens as ever
    (385, 1536, 3, 1), (1024, 1536, 3, 1), (1500, 1536, 3, 0),
    (385, 2048, 4, 1), (2048, 2048, 4, 1), (3000, 2048, 4, 1), (4096, 2048, 4, 0), (8192, 2048, 2, 0),
    (2048, 4096, 8, 1), (6000, 4096, 3, 1), (8192, 4096, 2, 0),
    (2048, 8192, 8, 1), (9472, 8192, 2, 1), (9473, 8192, 1, 0),                      # 75 tiles of 128 tokens: two shares are more than a round
])
def test_few_outputs_over_many_tokens_are_cut(lib, T, K, shares, bf16):
    """fp32 results wherever they can be cut, whose sums are the more exact for it; bf16 results where that is faster."""
    for N in (16, 64, 128):
        assert lib.zlm_gemm_tc_ksplit(T, N, K) == shares
        assert all(lib.zlm_gemm_tc_takes_few_form(T, N, K, m) == (T <= 384 or shares > 1) for m in (1, 2))
        assert all(lib.zlm_gemm_tc_takes_few_form(T, N, K, m) == bf16 for m in (0, 3, 7, 8))
        assert bf16 or lib.zlm_gemm_tc_mode_width(T, N, K, 0) == 128
    assert lib.zlm_gemm_tc_ksplit(max(T, 385), 129, K) == 1     # two tiles of outputs: never


@pytest.mark.parametrize("T,N,K,whole", [
    (1024, 1024, 704, 0), (1024, 1024, 768, 1), (385, 4096, 512, 0), (1024, 1024, 64, 0),         # pairs, tiles of 128 columns: from 12 stages
    (700, 8192, 1984, 0), (700, 8192, 2048, 1),                                                 # of 224: from 32
    (2048, 2048, 2048, 0), (2048, 24576, 3008, 0), (2048, 24576, 3072, 1),                      # of 256: from 48
    (143, 6144, 4096, 1), (300, 4096, 1024, 1), (300, 4096, 704, 0), (143, 2048, 2048, 0),      # stand-alone, two token tiles and more
    (17, 4096, 4096, 0), (64, 8192, 2048, 0), (100, 6144, 4096, 0), (128, 4096, 12288, 0),      # one: the weights come from memory
    (512, 128, 8192, 1), (2048, 128, 8192, 0), (4096, 128, 8192, 0),                                                  # few outputs over many tokens
    (300, 8192, 1536, 0), (300, 8192, 2048, 1),                                                 # persistent few-token blocks
])
def test_who_issues_a_product(lib, T, N, K, whole):
    assert lib.zlm_gemm_tc_issues_whole(T, N, K, 2) == whole


@pytest.mark.parametrize("T,N,hd,width", [
    (2048, 128, 128, 128), (2048, 128, 32, 128), (9472, 128, 128, 128),      # one head in all: half of a wide tile would be empty
    (2048, 512, 128, 128), (512, 4096, 128, 128), (512, 4096, 256, 256), (2048, 4096, 128, 256), (30000, 4096, 128, 256),
])
def test_projection_tile_width(lib, T, N, hd, width):
    assert lib.zlm_gemm_tc_qkv_width(T, N, hd) == width


def test_tcgen05_product_takes_what_tma_can_address(lib):
    assert lib.zlm_gemm_tc_supported(64, 4096, 4096, 4096) == 1
    assert lib.zlm_gemm_tc_supported(64, 4096, 4100, 4100) == 0      # rows of K elements must be 16-byte multiples
    assert lib.zlm_gemm_tc_supported(64, 4096, 4096, 4100) == 0


@pytest.mark.parametrize("T,N,K,width", [
    (2048, 4096, 4096, 240),     # 144 tiles of 240 on 74 pairs: two full rounds (128 of 256: the second 73 % full)
    (2048, 6144, 4096, 240),
    (2048, 24576, 4096, 256),    # 768 tiles: 11 rounds either way, the wide tile reuses the activations more
    (2048, 5120, 8192, 224),     # three rounds at every width: the narrowest of them
    (2048, 1024, 2048, 128),     # 32 tiles of 256 would leave more than half of the pairs idle
    (65143, 4096, 4096, 256),    # many rounds: the width hardly matters, so the widest
    (300, 4096, 4096, 0),        # few tokens: the other forms
])
def test_many_token_tile_width(lib, T, N, K, width):
    assert lib.zlm_gemm_tc_tile_width(T, N, K) == width


@pytest.mark.parametrize("T,N,K,modes,width", [
    (2048, 4096, 4096, (1, 2), 240), (2048, 4096, 4096, (0,), 256),          # bf16 rows are no whole boxes of 240 columns
    (2048, 6144, 4096, (1, 2), 240), (2048, 6144, 4096, (0,), 256),
    (2048, 5120, 8192, (0, 1, 2), 224),
    (512, 12288, 2048, (3, 7, 8), 224), (2048, 8192, 1024, (3, 7, 8), 224),  # gate and up: the rule whatever the boxes
    (385, 12288, 2048, (3, 7, 8), 224), (1500, 11008, 2048, (3, 7, 8), 240),
    (2048, 24576, 4096, (0, 1, 2, 3, 7, 8), 256), (512, 2048, 1024, (0, 1, 2, 3, 7, 8), 128),
])
def test_many_token_tile_width_by_what_leaves_the_tile(lib, T, N, K, modes, width):
    for mode in modes:
        assert lib.zlm_gemm_tc_mode_width(T, N, K, mode) == width


@pytest.mark.parametrize("R,max_new,nq,nkv,heads", [
    (1, 2048, 32, 8, 2),     # 256 blocks of two heads: enough for 148 SMs
    (1, 2048, 16, 8, 1),     # two heads per block would be 128 blocks, the longest twice as long
    (1, 8192, 16, 8, 2),     # long prompt: the spread work outweighs the longest block
    (1, 2048, 64, 8, 2),
    (1, 2048, 8, 8, 1),      # groups of one head
    (1, 2048, 24, 8, 1),     # odd groups
    (5, 300, 32, 8, 2),
    (64, 2048, 16, 8, 2),    # many prompts: plenty of blocks
])
def test_prefill_attention_heads_per_block(lib, R, max_new, nq, nkv, heads):
    assert lib.zlm_attention_prefill_tc_heads(R, max_new, nq, nkv) == heads


@pytest.mark.parametrize("rows,pages,want", [
    (8, 40, (7, 6)), (8, 48, (7, 7)), (8, 64, (7, 10)),        # 64 pairs: a part for every block the device holds
    (16, 64, (3, 22)), (24, 40, (2, 20)), (32, 64, (1, 64)), (48, 40, (1, 40)),   # but no second wave
    (1, 40, (10, 4)), (1, 64, (16, 4)), (1, 16, (8, 2)), (4, 64, (7, 10)),        # few pairs: fewer, longer parts
    (64, 40, (2, 24)), (64, 8, (1, 8)),                        # more pairs than the device holds: two waves
])
def test_decode_attention_cut(rows, pages, want):
    """The cut of the decode attention at 8 kv heads on a device that holds 444 blocks, as timed."""
    from zlm_b200.kernels import decode_splits
    splits, per = decode_splits(rows, 8, pages, 444)
    assert (splits, per) == want
    assert splits * per >= pages and (splits - 1) * per < pages      # the parts cover the pages, none is empty by design
    assert rows * 8 > 444 or splits * rows * 8 <= 444 * 1.1          # one wave of blocks wherever the pairs allow it


def test_decode_attention_cut_always_covers_the_pages():
    """Whatever the batch, the heads and the length: the parts cover every page, none of them is
    empty by design, and there are no more of them than the combine takes."""
    from zlm_b200.kernels import decode_splits
    for blocks in (444, 132 * 3, 8):
        for rows in (1, 2, 3, 4, 7, 8, 16, 17, 27, 28, 31, 32, 55, 56, 64, 200, 1024):
            for nkv in (1, 2, 5, 8, 16, 64):
                for pages in list(range(1, 70)) + [128, 500, 2048, 16384]:
                    splits, per = decode_splits(rows, nkv, pages, blocks)
                    assert per >= 1 and 1 <= splits <= 1024, (rows, nkv, pages, blocks, splits, per)
                    assert splits * per >= pages, (rows, nkv, pages, blocks, splits, per)
                    assert (splits - 1) * per < pages, (rows, nkv, pages, blocks, splits, per)


def test_latent_decode_splits_cover_the_pages():
    """The latent attention's cut of a decode step: splits x pages per split cover the longest sequence for
    every batch, head-tile count, length and wave, with at most 1024 splits, and one wave where that is possible."""
    from zlm_b200.kernels import latent_decode_splits
    for rows in (1, 2, 8, 17, 64, 300):
        for tiles in (1, 2, 8):
            for bucket in (1, 2, 3, 8, 32, 64, 512, 4096):
                for wave in (8, 148, 444, 2000):
                    splits, per = latent_decode_splits(rows, tiles, bucket, wave)
                    assert splits * per >= bucket and (splits - 1) * per < bucket and 1 <= splits <= 1024
                    if bucket >= 2 and splits <= 512:
                        assert per >= 2
                    if bucket * rows * tiles > 2 * wave and splits < 1024:
                        assert splits * rows * tiles <= wave + rows * tiles


@pytest.mark.parametrize("R,H,D,V,maxp,fits", [
    (1, 1, 128, 65536, 1, 1), (1, 2, 64, 128 * 65535, 2, 1), (1, 1, 1, 128 * 65535 + 1, 1, 0),        # 128 columns by 65,535
    (1 << 20, 16, 64, 128, 1, 1), (1 << 20, 32, 64, 128, 1, 0)])                                       # sequences x heads x rows
def test_linear_attention_takes_wide_heads(lib, R, H, D, V, maxp, fits):
    assert lib.zlm_linear_attention_fits(R, H, D, V, maxp) == fits


@pytest.mark.parametrize("R,max_new,takes", [(1, 1, 1), (65535, 1, 1), (65536, 1, 0), (1, 32 * 65535, 1), (1, 32 * 65535 + 1, 0)])
def test_32_bit_attention_leaves_what_its_tiles_cannot_number_to_single_queries(lib, R, max_new, takes):
    from ctypes import c_float
    assert lib.zlm_attention_f32_tile_supported(16, 4, 128, 2048, 2048, c_float(0.0), 1, 0, 0, R, max_new) == takes


@pytest.mark.parametrize("R,T,max_new,W,size", [
    (1, 2048, 2048, 2048, 8), (1, 8192, 8192, 4096, 8), (2, 1999, 1000, 1024, 8),           # one long sequence: the whole cluster
    (64, 8192, 128, 2048, 1), (16, 2048, 128, 4096, 1), (64, 191, 128, 2048, 1),             # many short ones: as few blocks as can be
    (64, 2111, 2048, 1024, 4), (21, 1824, 1024, 4096, 2), (1, 1, 1, 64, 1), (65535, 65535, 1, 8192, 1)])
def test_recurrent_units_clusters_by_rounds_and_blocks(lib, R, T, max_new, W, size):
    assert lib.zlm_rglru_cluster_size(R, T, max_new, W) == size


@pytest.mark.parametrize("T,R,units,hdp,taps,runs", [
    (2999, 3, 24, 128, 4, 1), (256, 1, 48, 128, 4, 1), (255, 1, 48, 128, 4, 0),
    (512, 1, 8, 128, 4, 0), (1152, 1, 8, 128, 4, 1), (256, 1, 24, 128, 4, 0),                  # warps of eight tokens that fill the GPU
    (4096, 4096, 48, 128, 4, 0), (320, 64, 24, 128, 4, 0), (512, 64, 24, 128, 4, 1),            # decode steps, and a prompt beside them
    (512, 256, 48, 128, 4, 0), (2048, 1024, 48, 128, 4, 1),                                     # two tokens a sequence
    (2999, 3, 24, 256, 4, 0), (2999, 3, 24, 128, 1, 0), (2999, 3, 24, 128, 6, 0)])
def test_convolution_in_runs_where_they_win(lib, T, R, units, hdp, taps, runs):
    assert lib.zlm_conv_runs(T, R, units, hdp, taps) == runs


@pytest.mark.parametrize("longest,R,H,D,V,columns", [
    (1, 16, 8, 64, 128, 1), (1, 8, 8, 64, 128, 0), (3, 64, 8, 64, 128, 1), (4, 64, 8, 64, 128, 0), (1, 64, 8, 64, 64, 0),
    (1, 8, 8, 128, 128, 1), (1, 4, 8, 128, 128, 0), (1, 4, 8, 128, 256, 1), (1, 64, 8, 32, 128, 0), (1, 96, 8, 32, 64, 1)])
def test_linear_attention_by_columns_where_sequences_and_heads_fill_the_gpu(lib, longest, R, H, D, V, columns):
    assert lib.zlm_linear_attention_by_columns(longest, R, H, D, V) == columns
