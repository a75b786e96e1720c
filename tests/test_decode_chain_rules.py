"""Which decoders may run the short decode chain (host code only): the library says what its projection kernel takes, so that a
step it refuses runs layer by layer instead of failing half way."""

import ctypes

import pytest
import torch

from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import backbone as BB


def check(T, in_dim, outs, r, S=4, n_buckets=5, aligned=True):
    n = len(outs)
    at = 4096 if aligned else 4098  # (host code: the pointers are looked at, never followed)
    slabs = (ctypes.c_void_p * n)(*[at] * n)
    widths, cols = (ctypes.c_int32 * n)(*outs), (ctypes.c_int32 * n)(*[sum(outs[:i]) for i in range(n)])
    return N.lib().lora_b200_decode_linear_check(T, in_dim, 4096, in_dim, sum(outs), n, slabs, slabs, widths, cols, S, r, n_buckets)


@pytest.mark.parametrize("r", range(16, 257, 16))
def test_ranks_of_a_cluster(r):
    assert check(64, 1024, [1024], r) == 0
    assert check(64, 1024, [4096, 4096], r) == 0
    # three slices stack 3 r rank rows, and a cluster of eight CTAs holds 512
    assert (check(64, 1024, [1024, 128, 128], r) == 0) == (3 * r <= 512)


def test_refused_forms():
    assert check(64, 1024, [1024], 24) != 0 and check(64, 1024, [1024], 272) != 0
    assert check(64, 1000, [1024], 32) != 0 and check(64, 1024, [1020], 32) != 0
    assert check(129, 1024, [1024], 32) != 0 and check(64, 1024, [1024], 32, n_buckets=0) != 0
    assert check(64, 1024, [1024], 32, aligned=False) != 0


@pytest.mark.parametrize("r,ok", [(16, True), (160, True), (176, False), (256, False), (24, False)])
def test_decoder_asks_the_library(r, ok):
    cfg = BB.DecoderConfig(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=128, num_layers=1,
                           max_position=64, max_loras=2, max_lora_rank=r)
    model = BB.Decoder(cfg).to(torch.bfloat16)
    assert model._chain_projections_ok(8, 3) == ok
    assert model._chain_projections_ok(8, None)  # without adapters
    assert not model._chain_projections_ok(8, 0)
