"""The decode kernel's cluster size (host code only): the rule takes every problem that some cluster size can run."""

import ctypes

import pytest

from nanovllm_voxcpm_b200 import _native as N


def chosen(T, in_dim, outs, r, n_buckets, dtype=N.DT_BF16, beside_gemm=0):
    widths = (ctypes.c_int32 * len(outs))(*outs)
    return N.lib().lora_b200_bucket_cluster(T, in_dim, len(outs), widths, r, n_buckets, dtype, beside_gemm)


@pytest.mark.parametrize("T, in_dim, outs, r, n_buckets", [
    (1024, 1024, [65536], 96, 1025),             # 1024 tiles of 64 columns, 256 of them a CTA at most: clusters of four
    (4096, 64, [65536], 32, 4097),               # 256 tiles in one CTA
    (4096, 64, [65536 + 256], 32, 4097),         # one more
    (4096, 1024, [32768, 32768], 256, 4097),     # tiles of 32 columns: eight
    (1000, 2048, [200000], 64, 2000),
])
def test_wide_outputs_get_a_cluster_that_holds_them(T, in_dim, outs, r, n_buckets):
    takes = []
    for c in (1, 2, 4, 8):
        N.set_option(N.OPT_CLUSTER, c)
        try:
            takes.append(chosen(T, in_dim, outs, r, n_buckets))
        finally:
            N.set_option(N.OPT_CLUSTER, 0)
    assert any(takes) and chosen(T, in_dim, outs, r, n_buckets) in takes


def test_refused_forms():
    assert chosen(8, 1024, [1024], 40, 8) == 0 and chosen(8, 1000, [1024], 32, 8) == 0
    assert chosen(8, 1024, [1024 * 1024], 256, 8) == 0 and chosen(8, 1024, [1024], 32, 0) == 0
    assert chosen(8, 1024, [1024], 32, 8, N.DT_F16, beside_gemm=1) == 0 and chosen(8, 1024, [1024], 32, 8, N.DT_F32) == 0
