"""The kernels for bucketed batches of both 16-bit types (``csrc/grouped_tc.cuh``, ``csrc/bgmv_fused.cuh``): parity with the
CPU oracle at the edges of their tiles - one token, 16- and 32-token chunks and their remainders, partial 128-row output
tiles, K tails and K parts, every rank, popular buckets, mixed ranks, slots of rank 0 - through ``lora_b200_add`` with the
kernel asked for by name."""

import ctypes
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from helpers import assert_lora_close
from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import workloads as W
from nanovllm_voxcpm_b200.lora_ops import LoRAKernelMeta, lora_expand, lora_shrink
from oracle import lora_oracle as O
from test_parity_gpu import metadata_for

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [
    # T, in, outs, S, r, kwargs
    (1, 1024, [1024, 128, 128], 4, 32, dict(p_none=0.0)),
    (17, 64, [8], 3, 16, dict()),
    (37, 1024, [1024], 16, 16, dict(p_none=0.25)),
    (63, 200, [136, 8, 40], 2, 32, dict()),                # K tail of 8 columns, slices of odd tile counts
    (64, 512, [4096], 1, 64, dict(p_none=0.0)),            # exactly one full chunk
    (65, 1792, [512, 512], 1, 64, dict(p_none=0.0)),       # one row in a second chunk
    (200, 4096, [1024], 5, 32, dict()),
    (301, 1024, [4096, 4096], 3, 32, dict()),              # several chunks per bucket
    (150, 2048, [2048, 256, 256], 12, 64, dict(ranks=[8, 16, 64] * 4)),
    (90, 320, [256, 128, 64, 72], 6, 16, dict(ranks=[16, 0, 3, 16, 8, 1])),
]


@pytest.mark.parametrize("cluster", [1, 4, 8])
@pytest.mark.parametrize("r", [64, 128, 256])
def test_fused_decode_kernel_wide_ranks(r, cluster):
    """Ranks whose output tiles are 128, 64 and 32 rows high (several tiles per step), clusters with few rank rows each."""
    p = W.make_projection(70 + r, 21, 2048, [1184, 96], 3, r)
    d = p.to_device(DEV)
    y = d.y.clone()
    N.set_option(N.OPT_CLUSTER, cluster)
    try:
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata_for(p.token_to_slot, "graph", 3), 1.0,
                        impl=N.IMPL_BGMV)
        torch.cuda.synchronize()
    finally:
        N.set_option(N.OPT_CLUSTER, 0)
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, p.token_to_slot, 1.0, p.col_offsets), max_abs=6e-2, what=f"r{r}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("cluster", [1, 2, 8])
@pytest.mark.parametrize("outs, r", [([160, 200, 72], 32), ([8, 296, 256, 264], 16), ([520, 40], 64), ([264, 32, 8], 48)])
def test_output_tiles_dealt_over_the_warps(outs, r, cluster, dtype):
    """Slices of partial tiles: a tile's rows begin at any warp and may run over the last one to the first."""
    p = W.make_projection(800 + r, 19, 1024, outs, 2, r, dtype=dtype)
    d = p.to_device(DEV)
    y = d.y.clone()
    N.set_option(N.OPT_CLUSTER, cluster)
    try:
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata_for(p.token_to_slot, "graph", 2), 1.0,
                        impl=N.IMPL_BGMV)
        torch.cuda.synchronize()
    finally:
        N.set_option(N.OPT_CLUSTER, 0)
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, p.token_to_slot, 1.0, p.col_offsets), what=f"{outs} r{r}")


@pytest.mark.parametrize("r, dtype", [(64, torch.float16), (128, torch.float16), (256, torch.float16), (48, torch.bfloat16), (80, torch.bfloat16)])
@pytest.mark.parametrize("cluster", [2, 8])
def test_a_warps_next_block_lies_several_tiles_ahead(r, dtype, cluster):
    """Adds and expands that read y (fp16, bf16 at ranks that are no multiple of 32, ``lora_expand``) where tiles are 128, 64 and 32 rows
    high: y of a warp's next block is asked for while it multiplies the one before, tiles of other warps lying between."""
    T, S, outs = 21, 3, [1184, 96, 8]
    p = W.make_projection(850 + r, T, 512, outs, S, r, dtype=dtype)
    d = p.to_device(DEV)
    y, y2 = d.y.clone(), d.y.clone()
    km = LoRAKernelMeta.make(S, T, DEV)
    km.prepare_tensors(d.token_to_slot)
    args = km.meta_args(T, specialize_active_lora=True)
    tmp = torch.zeros(len(outs), T, r, device=DEV, dtype=torch.float32)
    N.set_option(N.OPT_CLUSTER, cluster)
    try:
        # (three slices of 256 ranks make 96 rank rows a CTA in clusters of eight, the kernel takes 64: one slice less)
        k = 2 if r == 256 else 3
        LORA.launch_add(y, d.x, d.a_slabs[:k], d.b_slabs[:k], d.out_sizes[:k], d.col_offsets[:k], metadata_for(p.token_to_slot, "graph", S), 1.0,
                        impl=N.IMPL_BGMV)
        lora_shrink(d.x, d.a_slabs, tmp, *args, 1.0)
        lora_expand(tmp, d.b_slabs, y2, *args, offset_start=0, add_inputs=True)
        torch.cuda.synchronize()
    finally:
        N.set_option(N.OPT_CLUSTER, 0)
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.add_lora(p.y, p.x, p.a_slabs[:k], p.b_slabs[:k], p.token_to_slot, 1.0, p.col_offsets[:k]), what=f"add r{r}")
    assert_lora_close(y2, O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, p.token_to_slot, 1.0, p.col_offsets), what=f"expand r{r}")


@pytest.mark.parametrize("T, in_dim, outs, S, r, cluster", [
    (4, 6144, [2048], 8, 32, 8),           # eight CTAs although they lose the K split of six parts
    (4, 5120, [1280], 8, 32, 8),           # ... of five
    (4, 4096, [1024], 8, 32, 4),           # with the K split of four parts
    (37, 1024, [4096, 4096], 16, 16, 8),   # 16 rank rows
    (64, 1024, [1024], 48, 32, 4),         # by the clusters that fit
    (90, 1024, [1024], 100, 32, 2),
    (256, 1024, [1024], 300, 32, 1),
])
def test_fused_decode_kernel_with_the_cluster_it_chooses(T, in_dim, outs, S, r, cluster):
    widths = (ctypes.c_int32 * len(outs))(*outs)
    assert N.lib().lora_b200_bucket_cluster(T, in_dim, len(outs), widths, r, S + 1, N.DT_BF16, 0) == cluster
    p = W.make_projection(900 + T, T, in_dim, outs, S, r)
    d = p.to_device(DEV)
    y = d.y.clone()
    LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata_for(p.token_to_slot, "graph", S), 1.0,
                    impl=N.IMPL_BGMV)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, p.token_to_slot, 1.0, p.col_offsets), what=f"{T} {in_dim} {outs}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("impl", [N.IMPL_GROUPED, N.IMPL_BGMV], ids=["grouped", "bgmv"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_bucketed_kernels_match_oracle(case, impl, dtype):
    T, in_dim, outs, S, r, kw = CASES[case]
    if impl == N.IMPL_BGMV and in_dim % 32:
        pytest.skip("the fused decode kernel takes multiples of 32")
    p = W.make_projection(100 + case, T, in_dim, outs, S, r, dtype=dtype, **kw)
    d = p.to_device(DEV)
    scale = torch.linspace(0.5, 1.5, S)
    conv = ("eager", "graph", "vllm")[case % 3]
    y = d.y.clone()
    LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata_for(p.token_to_slot, conv, S), 0.5,
                    rank_per_slot=d.ranks, scale_per_slot=scale.to(DEV), impl=impl)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    b = [t.float() * scale.view(-1, 1, 1) for t in p.b_slabs]
    ref = O.add_lora(p.y, p.x, p.a_slabs, b, p.token_to_slot, 0.5, p.col_offsets)
    assert_lora_close(y, ref, what=f"{CASES[case]} {dtype}")
    none = p.token_to_slot < 0
    assert torch.equal(y.cpu()[none].view(torch.int16), p.y[none].view(torch.int16)), "rows without adapter changed"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", [0, 2, 5, 7, 8, 9])
def test_operators_with_bucket_arrays_match_oracle(case, dtype):
    """``lora_shrink`` and ``lora_expand`` with the vLLM-style arrays: intermediate in the activations' type and in fp32, rows
    without adapter zero, expand adding and overwriting."""
    T, in_dim, outs, S, r, kw = CASES[case]
    p = W.make_projection(300 + case, T, in_dim, outs, S, r, dtype=dtype, **kw)
    d = p.to_device(DEV)
    km = LoRAKernelMeta.make(S, T, DEV)
    km.prepare_tensors(d.token_to_slot)
    args = km.meta_args(T, specialize_active_lora=True)
    none = p.token_to_slot < 0
    for out_dtype in (dtype, torch.float32):
        tmp = torch.full((len(outs), T, r), 3.0, device=DEV, dtype=out_dtype)
        lora_shrink(d.x, d.a_slabs, tmp, *args, 0.5)
        ref_tmp = O.shrink(p.x, p.a_slabs, p.token_to_slot, 0.5)
        assert_lora_close(tmp, ref_tmp, what=f"shrink {out_dtype}")
        assert not tmp.cpu()[:, none].any()
        y = d.y.clone()
        lora_expand(tmp, d.b_slabs, y, *args, offset_start=0, add_inputs=True)
        assert_lora_close(y, O.expand(p.y, tmp.float().cpu(), p.b_slabs, p.token_to_slot), what="expand")
        assert torch.equal(y.cpu()[none].view(torch.int16), p.y[none].view(torch.int16))
        k = len(outs) - 1
        y2 = torch.zeros_like(d.y)
        lora_expand(tmp[k:].contiguous(), d.b_slabs[k:], y2, *args, offset_start=p.col_offsets[k], add_inputs=False)
        want = O.expand(torch.zeros_like(p.y), tmp[k:].float().cpu(), p.b_slabs[k:], p.token_to_slot, p.col_offsets[k], False)
        assert_lora_close(y2, want, what="expand, overwriting")
        assert not y2.cpu()[:, : p.col_offsets[k]].any()
    assert N.device_status(reset=True) == 0


@pytest.mark.parametrize("contiguous", [True, False], ids=["prompts", "scattered"])
def test_operators_choose_the_kernel_by_the_order_of_the_rows(contiguous):
    """Batches of prefill size, where each call launches a kernel for contiguous and one for scattered rows and one of them does
    the work: once, whatever the order."""
    T, outs, S, r = 1100, [2048, 2048, 2048], 4, 64
    slots = None
    if contiguous:
        slots = torch.repeat_interleave(torch.tensor([2, -1, 0, 3, 2], dtype=torch.int32), torch.tensor([300, 129, 1, 500, 170]))
    p = W.make_projection(400, T, 2048, outs, S, r, token_to_slot=slots)
    d = p.to_device(DEV)
    km = LoRAKernelMeta.make(S, T, DEV)
    km.prepare_tensors(d.token_to_slot)
    args = km.meta_args(T, specialize_active_lora=True)
    tmp = torch.full((3, T, r), 3.0, device=DEV, dtype=torch.bfloat16)
    lora_shrink(d.x, d.a_slabs, tmp, *args, 0.5)
    assert_lora_close(tmp, O.shrink(p.x, p.a_slabs, p.token_to_slot, 0.5), what="shrink")
    y = d.y.clone()
    lora_expand(tmp, d.b_slabs, y, *args, offset_start=0, add_inputs=True)
    assert_lora_close(y, O.expand(p.y, tmp.float().cpu(), p.b_slabs, p.token_to_slot), what="expand")
    none = p.token_to_slot < 0
    assert not tmp.cpu()[:, none].any()
    assert torch.equal(y.cpu()[none].view(torch.int16), p.y[none].view(torch.int16))
    assert N.device_status(reset=True) == 0


def test_auto_takes_the_grouped_kernels_with_the_scratch_that_the_query_names():
    """A batch over many large adapters: ``lora_b200_workspace_bytes`` of scratch is enough for the kernel that IMPL_AUTO
    chooses, and one that does not get what this batch needs runs on the fused decode kernel instead of failing."""
    T, in_dim, outs, S, r = 640, 14336, [4096], 60, 64
    p = W.make_projection(500, T, in_dim, outs, S, r, p_none=0.0)
    d = p.to_device(DEV)
    meta = metadata_for(p.token_to_slot, "graph", S)
    need = N.lib().lora_b200_grouped_workspace_bytes(T, in_dim, len(outs), r, S + 1)
    given = N.workspace_bytes(T, len(outs), r)
    assert need <= given

    def run(impl, nbytes):
        y, ws = d.y.clone(), torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, meta, 1.0, impl=impl, workspace=ws)
        torch.cuda.synchronize()
        assert N.device_status(reset=True) == 0
        return y

    grouped, fused = run(N.IMPL_GROUPED, need), run(N.IMPL_BGMV, need)
    assert torch.equal(run(N.IMPL_AUTO, given), grouped) and not torch.equal(grouped, fused)
    assert torch.equal(run(N.IMPL_AUTO, need - 1), fused)
    with pytest.raises(RuntimeError, match="scratch"):
        run(N.IMPL_GROUPED, need - 1)
    # one rounding of the sum to bf16 (and of the delta): outputs of size 4 to 8 have steps of 2^-5
    ref = O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, p.token_to_slot, 1.0, p.col_offsets)
    assert_lora_close(grouped, ref, max_abs=2 * ref.abs().max().item() * 2 ** -8, what="grouped")


def test_two_launch_kernels_on_two_streams_at_once():
    """Calls that keep an intermediate in the package's scratch, from two threads on streams of their own and then on one stream."""
    T, S, r, rounds = 96, 6, 64, 30
    p = [W.make_projection(600 + i, T, 2048, [2048], S, r, p_none=0.0) for i in range(2)]
    d = [q.to_device(DEV) for q in p]
    meta = [metadata_for(q.token_to_slot, "graph", S) for q in p]

    def run(i, stream):
        y = d[i].y.clone()
        with torch.cuda.stream(stream):
            stream.wait_stream(torch.cuda.default_stream())
            for _ in range(rounds):
                LORA.launch_add(y, d[i].x, d[i].a_slabs, d[i].b_slabs, d[i].out_sizes, d[i].col_offsets, meta[i], 0.01, impl=N.IMPL_GROUPED)
        stream.synchronize()
        return y

    streams = [torch.cuda.Stream() for _ in range(2)]
    want = [run(i, streams[i]) for i in range(2)]
    with ThreadPoolExecutor(2) as pool:
        for pair in (streams, [streams[0]] * 2):
            got = list(pool.map(run, range(2), pair))
            for i in range(2):
                assert torch.equal(got[i], want[i])
    assert N.device_status(reset=True) == 0
