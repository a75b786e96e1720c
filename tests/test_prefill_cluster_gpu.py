"""The one-launch prefill kernel (``csrc/prefill_cluster.cuh``) at the edges of its blocks and clusters: row counts around the
lines where the cluster size and the rows of a block change, ragged last blocks, K splits with a short last part, many runs in
a block (several passes), runs that end at block lines, blocks without any adapter, one to four slices, every rank."""

import pytest
import torch

from helpers import assert_lora_close
from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import workloads as W
from oracle import lora_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def by_runs(T, S, longest, seed):
    """Slots of rows in runs of 1 .. longest rows, every fifth run or so without adapter."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    while len(out) < T:
        slot = int(torch.randint(-S // 4 - 1, S, (1,), generator=gen).clamp(min=-1))
        out += [slot] * int(torch.randint(1, longest + 1, (1,), generator=gen))
    return torch.tensor(out[:T], dtype=torch.int32)


def metadata(slots):
    from nanovllm_voxcpm_b200 import batch_plan as BP

    ctx = BP.build_lora_context_from_slot_list(slots.tolist(), device=DEV)
    return LORA.LoRAMetadata(ctx.token_to_slot, ctx.token_indices_sorted_by_slot, ctx.active_slot_ids, ctx.num_tokens_per_slot,
                             ctx.slot_start_offsets, ctx.no_lora_flag, ctx.num_active_loras)


# T, in, outs, S, r, longest run (0: one run of all rows but a head without adapter)
CASES = [
    (1, 64, [64], 1, 16, 1),                     # one row, one K step
    (64, 1024, [128, 64], 3, 32, 9),             # one block of 64 rows, eight K parts
    (65, 192, [320], 3, 64, 70),                 # two blocks, two groups of columns
    (960, 2048, [256, 64, 64], 5, 64, 200),      # groups that straddle slices
    (961, 2048, [256, 64, 64], 5, 64, 30),       # ... more blocks, several passes a block
    (1920, 576, [640], 4, 32, 400),              # K parts of five and four steps
    (1921, 1024, [192, 192], 4, 32, 5),          # clusters of 4, blocks of 64, 40 runs a block
    (4225, 320, [512], 6, 16, 300),              # clusters of 2, ragged
    (9472, 128, [64, 64, 64, 64], 2, 64, 900),   # two groups of one CTA, four slices of rank 64
    (9473, 128, [256], 2, 32, 0),                # one CTA a block
    (300, 1024, [448, 128, 192], 5, 64, 60),     # three groups, of one and of two slices
    (900, 256, [1536, 1600], 4, 32, 200),        # nine groups, the last one narrower
    (130, 64, [320, 64, 512, 128], 4, 64, 9),    # sixteen groups of one CTA, a tile each
    (300, 64, [4032], 3, 16, 7),                 # 21 groups, many runs a block
    (700, 1024, [1024, 128, 128], 6, 64, 150),   # ten groups of columns
    (2100, 1024, [1024, 128, 128], 4, 64, 40),   # rank rows of three slices in a block: partial sums where the K loop's ring was
]


@pytest.mark.parametrize("overwrite", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_prefill_add_matches_oracle(case, overwrite):
    T, in_dim, outs, S, r, longest = CASES[case]
    slots = by_runs(T, S, longest, case) if longest else torch.cat([torch.full((300,), -1), torch.zeros(T - 300)]).to(torch.int32)
    slots[0] = 0
    if T > 1000:
        slots[200:460] = -1  # at least one block without any adapter
    p = W.make_projection(700 + case, T, in_dim, outs, S, r, token_to_slot=slots)
    d = p.to_device(DEV)
    LORA.launch_add(d.y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=N.IMPL_SGMV, overwrite=overwrite)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    base = torch.full_like(p.y, -0.0) if overwrite else p.y
    # one 16-bit rounding of the intermediate, one of the delta, one of the sum: the tolerance stated for the path
    assert_lora_close(d.y, O.add_lora(base, p.x, p.a_slabs, p.b_slabs, slots, 0.5, p.col_offsets), what="prefill add")
    none = slots < 0
    assert torch.equal(d.y.cpu()[none].view(torch.int16), base[none].view(torch.int16)), "rows without adapter keep their bits"


@pytest.mark.parametrize("overwrite", [False, True])
def test_auto_needs_no_scratch_for_the_one_launch_kernel(overwrite):
    T, in_dim, outs, S, r = 1300, 1024, [1024, 128, 128], 4, 64
    slots = torch.arange(T, dtype=torch.int32) // 400
    p = W.make_projection(720, T, in_dim, outs, S, r, token_to_slot=slots)
    d = p.to_device(DEV)
    none = torch.empty(0, dtype=torch.uint8, device=DEV)

    def run(impl, workspace=None):
        y = d.y.clone()
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=impl, overwrite=overwrite,
                        workspace=workspace)
        torch.cuda.synchronize()
        assert N.device_status(reset=True) == 0
        return y

    prefill, bucket = run(N.IMPL_SGMV), run(N.IMPL_BGMV)
    assert torch.equal(run(N.IMPL_AUTO, none), prefill) and not torch.equal(prefill, bucket)
    with pytest.raises(RuntimeError, match="scratch"):
        run(N.IMPL_SGMV, none)


@pytest.mark.parametrize("T, in_dim, outs, r, prefill", [
    (2000, 1024, [1024, 128, 128], 32, False), (2500, 1024, [1024, 128, 128], 32, True),   # 35 and 44 MB of adapters for the bucket kernel
    (400, 2048, [2048, 256, 256], 64, False), (480, 2048, [6144, 6144], 64, True),         # 28 and 63 MB, fewer than 512 rows
    (1000, 1024, [4096, 4096], 16, False), (1300, 1024, [4096, 4096], 16, True),           # rank 16: as before up to 1184 rows
    (1300, 1024, [1024], 16, False), (3840, 256, [256], 32, False), (3841, 256, [256], 32, True),
])
def test_auto_takes_the_kernel_of_the_line(T, in_dim, outs, r, prefill):
    slots = torch.arange(T, dtype=torch.int32) * 4 // T
    p = W.make_projection(740, T, in_dim, outs, 4, r, token_to_slot=slots)
    d = p.to_device(DEV)

    def run(impl):
        y = d.y.clone()
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=impl)
        torch.cuda.synchronize()
        assert N.device_status(reset=True) == 0
        return y

    by_name = {True: run(N.IMPL_SGMV), False: run(N.IMPL_BGMV)}
    assert not torch.equal(by_name[True], by_name[False])
    assert torch.equal(run(N.IMPL_AUTO), by_name[prefill])


def test_auto_overwrites_with_the_prefill_kernel_at_rank_16():
    """1300 rows: an add of this size is the bucket kernel's, which cannot overwrite at rank 16."""
    T, outs = 1300, [1024]
    slots = torch.arange(T, dtype=torch.int32) * 4 // T
    p = W.make_projection(750, T, 1024, outs, 4, 16, token_to_slot=slots)
    d = p.to_device(DEV)
    y = [d.y.clone(), d.y.clone()]
    for out, impl in zip(y, (N.IMPL_AUTO, N.IMPL_SGMV)):
        LORA.launch_add(out, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=impl, overwrite=True)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0 and torch.equal(*y)


# T, in, outs, S, r, longest run: fused linears of the kernel (the plan's lines: one tile a CTA, one more over 1024 columns of x)
LINEAR = [
    (7, 64, [48], 2, 16, 3),                     # less than a tile of columns, some CTAs without any
    (333, 1024, [1024, 128, 128], 4, 32, 90),    # 1280 columns over eight CTAs
    (517, 4096, [208, 112], 3, 32, 4),           # slices of 16-column units, 40 runs a block, many passes
    (961, 320, [1000 - 8], 3, 64, 300),          # ragged columns, blocks of 72 rows
    (2200, 1024, [640, 640], 4, 64, 500),        # clusters of 4, two tiles a CTA
    (4300, 128, [512], 4, 16, 128),              # clusters of 2
    (517, 1024, [320], 3, 16, 4),                # many passes, CTAs that own no rank columns
    (70, 512, [1024, 320, 192], 3, 64, 20),      # groups of columns, of one to three slices
    (40, 2048, [960, 960], 4, 32, 9),            # four groups, a tile of 64 columns a CTA, seven stages
    (200, 1024, [2048, 1088], 4, 32, 60),        # four groups, the last one narrower
    (64, 1024, [1008], 2, 16, 0),                # ragged columns, partial sums of one piece
]


@pytest.mark.parametrize("case", range(len(LINEAR)))
def test_linear_of_the_cluster_kernel_matches_oracle(case):
    T, in_dim, outs, S, r, longest = LINEAR[case]
    slots = by_runs(T, S, longest, 50 + case) if longest else torch.ones(T, dtype=torch.int32)
    slots[0] = 0
    p = W.make_projection(800 + case, T, in_dim, outs, S, r, token_to_slot=slots, with_weight=True)
    d = p.to_device(DEV)
    bias = torch.randn(sum(outs), generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV)
    y = LORA.linear_lora(d.x, d.weight, bias, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, d.token_to_slot, 1.0)
    plain = LORA.linear_lora(d.x, d.weight, bias, [], [], [], [], None, 1.0)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    ref = O.linear_lora(p.x, p.weight, bias.cpu(), p.a_slabs, p.b_slabs, p.col_offsets, slots)
    # half a unit in the last place of the largest output, on top of the path's tolerance
    assert_lora_close(y, ref, max_abs=2e-2 + 2.0 ** -8 * float(ref.abs().max()), what="cluster linear")
    none = slots < 0
    assert torch.equal(y.cpu()[none].view(torch.int16), plain.cpu()[none].view(torch.int16)), "rows without adapter are the plain linear"


# T, in, outs, r, longest run: eight K parts; the place of the partial sums is written again by every pass of a block (and by every
# part of one)
REPEATED = [
    (995, 4096, [1024], 64, 5),                  # adds: sums where the K loop's ring was
    (197, 2048, [2048, 256, 256], 32, 4),
    (300, 2048, [1024], 32, 3),
    (412, 1024, [1024, 128, 128], 64, 6),        # fused linear: rank rows in two parts a pass
    (333, 1024, [1024, 128, 128], 32, 5),
]


@pytest.mark.parametrize("case", range(len(REPEATED)))
def test_partial_sums_of_many_passes_are_the_same_every_time(case):
    T, in_dim, outs, r, longest = REPEATED[case]
    linear = case >= 3
    slots = by_runs(T, 9, longest, 90 + case)
    slots[0] = 0
    p = W.make_projection(900 + case, T, in_dim, outs, 9, r, token_to_slot=slots, with_weight=linear)
    d = p.to_device(DEV)
    meta = metadata(slots)

    def run():
        if linear:
            return LORA.linear_lora(d.x, d.weight, None, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, d.token_to_slot, 1.0)
        y = d.y.clone()
        LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, meta, 1.0, impl=N.IMPL_SGMV)
        return y

    got = [run() for _ in range(30)]
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    for y in got[1:]:
        assert torch.equal(y.view(torch.int16), got[0].view(torch.int16))
    ref = (O.linear_lora(p.x, p.weight, None, p.a_slabs, p.b_slabs, p.col_offsets, slots) if linear
           else O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, slots, 1.0, p.col_offsets))
    # half a unit in the last place of the largest output, on top of the path's tolerance
    assert_lora_close(got[0], ref, max_abs=2e-2 + 2.0 ** -8 * float(ref.abs().max()), what="many passes")


@pytest.mark.parametrize("overwrite", [False, True])
@pytest.mark.parametrize("T, in_dim, outs, r", [(4300, 128, [1024, 256], 32), (4290, 192, [1024, 192], 16), (4736, 128, [640], 64)])
def test_two_ctas_take_an_odd_number_of_tiles_by_range(T, in_dim, outs, r, overwrite):
    """Clusters of two whose CTAs have 640 columns each (the second 640, 576), or 320: tiles of 256, 256, 128 and of 192, 128."""
    slots = by_runs(T, 4, 700, 60)
    slots[0] = 0
    p = W.make_projection(760, T, in_dim, outs, 4, r, token_to_slot=slots)
    d = p.to_device(DEV)
    LORA.launch_add(d.y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 1.0, impl=N.IMPL_SGMV, overwrite=overwrite)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    base = torch.full_like(p.y, -0.0) if overwrite else p.y
    assert_lora_close(d.y, O.add_lora(base, p.x, p.a_slabs, p.b_slabs, slots, 1.0, p.col_offsets), what="by range")
