"""The decode kernel's cluster size (host code only): the rule takes every problem that some cluster size can run, and the sizes
that measured fastest where it says so."""

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


# rows, input width, slices, rank, buckets, beside a GEMM; us a launch with clusters of 1 / 2 / 4 / 8, measured on a B200
MEASURED = [
    (8, 1024, [4096, 4096], 16, 33, 0, (16.3, 9.1, 5.4, 3.8)),
    (64, 1024, [1024], 32, 33, 0, (3.9, 2.8, 2.5, 3.7)),
    (128, 1024, [4096, 4096], 32, 129, 0, (20.2, 12.8, 15.1, 19.5)),
    (384, 1024, [1024], 32, 129, 0, (5.2, 5.0, 8.0, 16.8)),
    (4, 4096, [1024], 32, 9, 0, (9.5, 4.9, 3.1, 3.3)),
    (4, 5120, [1280], 32, 9, 0, (11.9, 7.3, 5.5, 3.7)),   # eight CTAs lose the K split of 5, 6 and 7 parts and are faster
    (4, 6144, [2048], 32, 9, 0, (14.9, 7.7, 5.5, 4.1)),
    (1, 7168, [1792], 32, 9, 0, (16.7, 9.6, 5.4, 4.4)),
    (128, 6144, [2048], 32, 9, 0, (15.4, 8.0, 6.1, 7.3)),
    (384, 2048, [6144, 6144], 32, 33, 0, (28.5, 21.8, 12.3, 16.3)),
    (256, 6144, [2048], 64, 33, 0, (35.3, 24.8, 16.4, 12.5)),
    (64, 2048, [6144, 6144], 64, 33, 0, (35.1, 34.6, 17.7, 11.9)),
    (4, 4096, [14336, 14336], 32, 9, 0, (54.2, 30.0, 15.8, 7.8)),
    (64, 1024, [1024, 128, 128], 32, 65, 1, (11.4, 11.4, 15.9, 26.1)),
    (64, 1024, [1024], 32, 65, 1, (6.7, 6.1, 9.9, 17.6)),
    (64, 1024, [4096, 4096], 32, 65, 1, (22.1, 15.0, 17.9, 23.7)),
    (64, 4096, [1024], 32, 65, 1, (13.4, 9.5, 13.9, 24.5)),
    (24, 1024, [4096, 4096], 32, 129, 1, (18.7, 11.7, 10.6, 13.9)),
    (8, 1024, [1024, 128, 128], 32, 33, 1, (8.8, 8.6, 7.9, 7.1)),
    (128, 1024, [1024], 32, 129, 1, (8.2, 11.4, 17.9, 35.5)),
    (24, 6144, [2048], 64, 33, 1, (36.3, 25.3, 17.9, 13.1)),
]


@pytest.mark.parametrize("T, in_dim, outs, r, n_buckets, beside_gemm, us", MEASURED)
def test_chosen_size_is_the_one_that_measured_fastest(T, in_dim, outs, r, n_buckets, beside_gemm, us):
    took = us[(1, 2, 4, 8).index(chosen(T, in_dim, outs, r, n_buckets, beside_gemm=beside_gemm))]
    assert took <= 1.02 * min(us)
