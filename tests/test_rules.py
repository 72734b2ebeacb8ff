"""The rules by which a call is given to one kernel or cut in one way, as far as the sizes decide."""

from __future__ import annotations

import ctypes

import pytest


def library():
    from litinfer_b200 import kernels
    return kernels.library()


def plan(M, N, K, deep=None):
    splits, cluster = ctypes.c_int(), ctypes.c_int()
    assert library().li_gemv_tcgen05_plan(M, N, K, ctypes.byref(splits), ctypes.byref(cluster), None if deep is None else ctypes.byref(deep)) == 0
    return splits.value, cluster.value


@pytest.mark.parametrize("N", [128, 512, 1536, 2048, 3584, 8192, 9472, 12288])
@pytest.mark.parametrize("K", [64, 4096, 8960, 18944])
def test_splits_of_the_streaming_product(N, K):
    """The token tile decides, not the tokens; one cluster a tile from 17 tokens on; whole clusters."""
    for counts in ((1, 7, 16), (17, 25, 32), (33, 64)):
        plans = {plan(M, N, K) for M in counts}
        assert len(plans) == 1
        splits, cluster = plans.pop()
        assert 1 <= splits <= max(1, K // 64) and splits % cluster == 0 and cluster <= 8
        if counts[0] > 16:
            assert splits == cluster


def test_splits_are_few_enough_for_one_cluster():
    """Eight for few tiles, or up to 28 with a long k; four or three where those are about a wave of CTAs."""
    assert [plan(8, 128 * t, 4096)[0] for t in (1, 18, 19, 37, 38, 49, 50, 60, 61, 74, 75)] == [8, 8, 4, 4, 3, 3, 4, 4, 2, 2, 1]
    assert [plan(8, 128 * t, 7168)[0] for t in (19, 28, 29)] == [8, 8, 4]
    assert plan(8, 1536, 512)[0] == 4                     # two k-blocks a CTA at least


@pytest.mark.gpu
@pytest.mark.parametrize("M", [32, 64])
def test_pipeline_depth_of_the_streaming_product(M):
    """Six stages where every CTA has a multiprocessor to itself, fewer where the CTAs come in waves or the clusters do not all fit."""
    import torch

    torch.zeros(1, device="cuda")

    def deep(N, K=8960):
        d = ctypes.c_int()
        plan(M, N, K, d)
        return d.value

    assert deep(128 * 148, 3584) == 1 and deep(128 * 149, 3584) == 0
    assert deep(1536) == 1 and deep(5120) == 1 and deep(8192) == 1
    # 16 clusters of eight: a B200 holds 15 of them with a multiprocessor a CTA
    assert plan(M, 2048, 8960) == (8, 8) and deep(2048) == 0


@pytest.mark.parametrize("tiles,M,N", [(119, 1792, 4352), (120, 2048, 3840), (128, 900, 8192), (144, 2304, 4096), (148, 1024, 9472), (150, 2560, 3840), (256, 2048, 8192)])
def test_which_products_the_persistent_kernel_takes(tiles, M, N):
    """From 120 tiles of 256 x 256 on; up to 148, which single CTAs do in one wave, only with less than 8,192 columns of k."""
    assert -(-M // 256) * -(-N // 256) == tiles
    for K in (1536, 4160, 8128, 8192, 13824):
        assert library().li_tcgen05_takes_persistent(M, N, K) == (tiles >= 120 and (tiles > 148 or K < 8129))


@pytest.mark.parametrize("heads,K,taken", [(6, 4096, 0), (18, 4096, 0), (10, 8128, 0), (20, 4096, 1), (20, 4032, 0), (24, 3072, 1), (24, 3008, 0), (23, 3072, 0), (36, 3584, 1),
                                           (96, 256, 1), (95, 256, 0)])
def test_which_q_k_v_of_few_tokens_the_tcgen05_kernel_takes(heads, K, taken):
    """Few heads stay on the register-fed kernel however long their rows are (more than 32 tokens: up to 8,192 columns)."""
    for T in (1, 32, 33, 64):
        assert library().li_rope_takes_tcgen05(T, heads * 128, K) == taken
    assert library().li_rope_takes_tcgen05(33, heads * 128, 8192) == 1
    assert library().li_rope_takes_tcgen05(32, heads * 128, 8192) == (heads >= 20)


def test_blocks_that_share_a_token_in_float32_attention():
    """As many as one wave has room for: 148 with heads of more than 64 elements, 296 with smaller ones."""
    def blocks(T, nh, nkv, dh):
        return library().li_attention_f32_blocks(T, nh, nkv, dh)

    assert [blocks(T, 12, 2, 128) for T in (1, 9, 10, 18, 19, 37, 38, 2048)] == [8, 8, 4, 4, 2, 2, 1, 1]
    assert [blocks(T, 32, 1, 64) for T in (9, 10, 18, 19, 37, 38)] == [8, 4, 4, 2, 2, 1]          # 32 heads: four parts
    assert blocks(16, 28, 4, 128) == 2


@pytest.mark.parametrize("M,N,K,taken", [(640, 7168, 5120, 1), (640, 27648, 5120, 1), (640, 5120, 5120, 1), (320, 37888, 3584, 1), (1536, 3584, 18944, 1),
                                         (2048, 7168, 5120, 1), (2048, 1536, 1536, 1), (2048, 17920, 1536, 0), (1024, 37888, 3584, 0), (128, 37888, 3584, 0),
                                         (640, 1536, 8960, 0), (256, 2048, 1536, 0)])
def test_which_products_have_their_tokens_as_columns(M, N, K, taken):
    """Where the padding of 256 tokens or half-empty waves cost more than the narrower tiles; never where k is split."""
    assert library().li_tcgen05_takes_tokens(M, N, K) == taken
