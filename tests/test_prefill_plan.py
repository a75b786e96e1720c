"""What the prefill kernels run for a batch (``lora_b200_prefill_plan``, host code), and every form of a split and every kernel of a
fused linear against the oracle at sizes for which the library says that it is the one that runs."""

import ctypes

import pytest
import torch

from helpers import assert_lora_close
from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import workloads as W
from oracle import lora_oracle as O

DEV = "cuda:0"
ADD, LINEAR, SILU = 0, 1, 2
CLUSTER, PAIRS, TILES = 1, 2, 3


def plan(T, in_dim, outs, r, form):
    """(kernel, CTAs of a cluster, groups of columns, rows of a block, tiles of a CTA, runs of a pass, exchanges of a pass, stages, most
    runs of a pass whose partial sums lie beside the K loop's ring)"""
    widths, split = (ctypes.c_int32 * len(outs))(*outs), (ctypes.c_int32 * 8)()
    return (N.lib().lora_b200_prefill_plan(T, in_dim, len(outs), widths, r, form, split), *split)


def by_runs(T, S, longest, seed):
    """Slots of rows in runs of 1 .. longest rows, every fifth run or so without adapter."""
    gen = torch.Generator().manual_seed(seed)
    out = [0]
    while len(out) < T:
        slot = int(torch.randint(-S // 4 - 1, S, (1,), generator=gen).clamp(min=-1))
        out += [slot] * int(torch.randint(1, longest + 1, (1,), generator=gen))
    return torch.tensor(out[:T], dtype=torch.int32)


def metadata(slots):
    from nanovllm_voxcpm_b200 import batch_plan as BP

    ctx = BP.build_lora_context_from_slot_list(slots.tolist(), device=DEV)
    return LORA.LoRAMetadata(ctx.token_to_slot, ctx.token_indices_sorted_by_slot, ctx.active_slot_ids, ctx.num_tokens_per_slot,
                             ctx.slot_start_offsets, ctx.no_lora_flag, ctx.num_active_loras)


def test_refused_forms():
    for form in (ADD, LINEAR, SILU):
        assert plan(300, 1000, [1024], 32, form)[0] == 0 and plan(300, 1024, [1024], 48, form)[0] == 0
        assert plan(0, 1024, [1024], 32, form)[0] == 0 and plan(300, 1024, [0], 32, form)[0] == 0
        assert plan(300, 1024, [1020], 32, form)[0] == 0
    assert plan(300, 1024, [1024], 32, 3)[0] == 0
    assert plan(300, 1024, [1000], 32, ADD)[0] == TILES     # no 64-column units: shrink and expand
    assert plan(300, 1024, [1000], 32, LINEAR)[0] != CLUSTER and plan(300, 1024, [1024, 1024], 32, SILU)[0] == PAIRS


def test_a_split_is_resident_and_covers_the_problem():
    resident = {1: 148, 2: 74, 4: 33, 8: 15}
    for form in (ADD, LINEAR):
        for T in (1, 63, 64, 65, 300, 511, 960, 961, 1920, 1921, 2112, 4224, 4225, 4736, 4737, 8000, 9472, 9473, 18944):
            for in_dim in (64, 192, 1024, 2048, 6144):
                for outs in ([64], [1024, 128, 128], [4096, 4096], [6144, 6144]):
                    for r in (16, 32, 64):
                        kernel, ck, groups, bm, tiles, runs, exchanges, stages, _ = plan(T, in_dim, outs, r, form)
                        if kernel != CLUSTER:
                            assert form == LINEAR and kernel in (PAIRS, TILES)
                            continue
                        blocks = -(-T // bm)
                        assert 64 <= bm <= 128 and bm % 8 == 0 and 1 <= runs <= 4 and exchanges >= 1 and stages >= 2 and tiles >= 1
                        assert blocks * groups <= resident[ck] or (ck == 1 and groups == 1 and bm == 128)
                        assert (in_dim // 64 + ck - 1) // ck * (ck - 1) < in_dim // 64  # every K part has a step


@pytest.mark.parametrize("T, in_dim, outs, split", [
    (4225, 1024, [4096, 4096], (2, 1, 64)), (4736, 2048, [6144, 6144], (2, 1, 64)), (4500, 4096, [3584, 3584], (2, 1, 64)),
    (4300, 1024, [4096], (2, 2, 120)), (4736, 1024, [4096], (2, 2, 128)),   # y of less than half of the L2
    (4737, 1024, [4096, 4096], (2, 1, 72)),                                  # one 64-row block more than clusters of two
])
def test_wide_outputs_of_as_many_blocks_as_clusters_of_two(T, in_dim, outs, split):
    assert plan(T, in_dim, outs, 64, ADD)[:4] == (CLUSTER, *split)


@pytest.mark.parametrize("T, in_dim, outs, kernel", [
    (3700, 4096, [1024], CLUSTER), (8000, 4096, [512], CLUSTER),          # a tile a CTA
    (3700, 2048, [2048], CLUSTER), (9000, 2048, [1024], CLUSTER),         # two, no more than the others have
    (1700, 4096, [4096], PAIRS), (3700, 4096, [2048], PAIRS), (6000, 4096, [1024], PAIRS), (12000, 4096, [512], TILES),  # two over 4096 columns
    (2000, 2048, [6144, 6144], PAIRS), (1000, 6144, [2048], TILES),
])
def test_kernel_of_a_fused_linear(T, in_dim, outs, kernel):
    assert plan(T, in_dim, outs, 32, LINEAR)[0] == kernel


# T, in, outs, S, r, longest run; kernel, CTAs of a cluster, groups, rows of a block
ADDS = [
    (960, 1024, [1024], 5, 32, 9, (CLUSTER, 8, 1, 64)),               # fifteen clusters of eight, several passes a block
    (995, 4096, [256], 5, 64, 9, (CLUSTER, 8, 1, 72)),                # ... four runs a pass: partial sums where the ring was
    (130, 1024, [1024], 4, 32, 7, (CLUSTER, 8, 2, 64)),               # eight CTAs, two groups, three blocks
    (200, 1024, [3072, 3072], 4, 64, 30, (CLUSTER, 8, 2, 64)),        # ... two tiles a CTA, a slice each
    (1990, 1024, [256, 64, 64], 4, 32, 40, (CLUSTER, 4, 1, 64)),      # ... four CTAs, three slices
    (7400, 512, [256, 64, 64], 4, 64, 200, (CLUSTER, 2, 1, 104)),     # sums of three slices never have a place of their own
]


def test_partial_sums_where_the_ring_was():
    assert plan(995, 4096, [256], 64, ADD)[8] < plan(995, 4096, [256], 64, ADD)[5] == 4
    assert plan(7400, 512, [256, 64, 64], 64, ADD)[8] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("overwrite", [False, True])
@pytest.mark.parametrize("case", range(len(ADDS)))
def test_add_of_a_split_matches_oracle(case, overwrite):
    T, in_dim, outs, S, r, longest, expected = ADDS[case]
    assert plan(T, in_dim, outs, r, ADD)[:4] == expected
    slots = by_runs(T, S, longest, 200 + case)
    p = W.make_projection(960 + case, T, in_dim, outs, S, r, token_to_slot=slots)
    d = p.to_device(DEV)
    LORA.launch_add(d.y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=N.IMPL_SGMV, overwrite=overwrite)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    base = torch.full_like(p.y, -0.0) if overwrite else p.y
    assert_lora_close(d.y, O.add_lora(base, p.x, p.a_slabs, p.b_slabs, slots, 0.5, p.col_offsets), what="add")
    none = slots < 0
    assert torch.equal(d.y.cpu()[none].view(torch.int16), base[none].view(torch.int16)), "rows without adapter keep their bits"


# T, in, outs, S, r, longest run; kernel, CTAs of a cluster, groups, rows of a block, tiles of a CTA; exchanges of a pass
LINEARS = [
    (2000, 256, [1024, 128, 128], 4, 16, 25, (CLUSTER, 4, 1, 64, 2), 1),   # four K parts
    (3000, 256, [2048, 1088], 4, 32, 40, (CLUSTER, 4, 1, 96, 4), 1),
    (2000, 512, [2048, 1088], 4, 64, 60, (CLUSTER, 4, 2, 128, 2), 2),
    (4000, 256, [1024, 128, 128], 4, 64, 90, (CLUSTER, 4, 1, 128, 2), 3),  # rank rows in three parts
    (1500, 512, [2048, 1088], 4, 16, 30, (CLUSTER, 8, 1, 104, 2), 1),      # eight
    (1500, 512, [2048, 1088], 4, 64, 50, (CLUSTER, 8, 1, 104, 2), 2),
    (700, 1024, [2048, 1088], 4, 64, 20, (CLUSTER, 8, 2, 104, 1), 2),
    (517, 512, [1024, 128, 128], 4, 64, 6, (CLUSTER, 8, 1, 64, 1), 2),
    (4000, 128, [1024, 128, 128], 4, 64, 90, (CLUSTER, 2, 1, 64, 3), 2),   # two
    (2300, 128, [2048, 1088], 4, 64, 50, (CLUSTER, 1, 7, 112, 2), 2),      # one
]


def check_linear(p, d, slots):
    bias = torch.randn(sum(p.out_sizes), generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    y = LORA.linear_lora(d.x, d.weight, bias.to(DEV), d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, d.token_to_slot, 1.0)
    plain = LORA.linear_lora(d.x, d.weight, bias.to(DEV), [], [], [], [], None, 1.0)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    ref = O.linear_lora(p.x, p.weight, bias, p.a_slabs, p.b_slabs, p.col_offsets, slots)
    # half a unit in the last place of the largest output, on top of the path's tolerance
    assert_lora_close(y, ref, max_abs=2e-2 + 2.0 ** -8 * float(ref.abs().max()), what="linear")
    none = slots < 0
    assert torch.equal(y.cpu()[none].view(torch.int16), plain.cpu()[none].view(torch.int16)), "rows without adapter are the plain linear"


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(LINEARS)))
def test_linear_of_a_split_matches_oracle(case):
    T, in_dim, outs, S, r, longest, expected, exchanges = LINEARS[case]
    got = plan(T, in_dim, outs, r, LINEAR)
    assert got[:5] == expected and got[6] == exchanges
    slots = by_runs(T, S, longest, 300 + case)
    p = W.make_projection(980 + case, T, in_dim, outs, S, r, token_to_slot=slots, with_weight=True)
    check_linear(p, p.to_device(DEV), slots)


def runs(lens, slots):
    return torch.repeat_interleave(torch.tensor(slots, dtype=torch.int32), torch.tensor(lens))


# T, in, outs, S, r, slots (None: independent rows, a run of almost every row); kernel behind the shrink
BEHIND_A_SHRINK = [
    (1409, 512, [4096, 224], 4, 64, runs([255, 2, 127, 1, 1024], [3, 0, 1, -1, 2]), PAIRS),
    (1793, 512, [4096, 224], 2, 32, runs([1792, 1], [1, 0]), PAIRS),
    (2300, 512, [2080, 32, 1024, 64], 3, 64, runs([128, 128, 300, 84, 896, 764], [0, 1, 2, -1, 0, 1]), PAIRS),
    (2700, 512, [4096], 6, 16, None, PAIRS),
    (2000, 320, [6144, 2080, 32], 5, 16, None, PAIRS),
    (500, 2048, [1024, 128, 128], 5, 64, runs([131, 3, 250, 100, 16], [4, -1, 0, 2, 3]), TILES),
    (700, 2048, [4000, 40], 4, 32, None, TILES),       # slices that end inside 16 columns: the delta in a launch of its own
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(BEHIND_A_SHRINK)))
def test_linear_behind_a_shrink_matches_oracle(case):
    T, in_dim, outs, S, r, slots, kernel = BEHIND_A_SHRINK[case]
    assert plan(T, in_dim, outs, r, LINEAR)[0] == kernel
    p = W.make_projection(520 + case, T, in_dim, outs, S, r, token_to_slot=slots, with_weight=True)
    check_linear(p, p.to_device(DEV), p.token_to_slot)


# T, in, outs, S, r; form: independent rows, so that a block holds rows of every slot in any order
SCATTERED = [
    (64, 1024, [128, 64], 9, 32, ADD), (128, 256, [512], 128, 16, ADD), (333, 512, [256, 64, 64], 8, 64, ADD), (300, 192, [4032], 2, 32, ADD),
    (4300, 128, [320], 5, 16, ADD),
    (40, 512, [320], 6, 32, LINEAR), (517, 512, [1024, 128, 128], 9, 64, LINEAR), (1500, 512, [2048, 1088], 40, 16, LINEAR),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(SCATTERED)))
def test_rows_of_a_slot_need_not_lie_together(case):
    T, in_dim, outs, S, r, form = SCATTERED[case]
    assert plan(T, in_dim, outs, r, form)[0] == CLUSTER
    slots = torch.randint(-1, S, (T,), generator=torch.Generator().manual_seed(case), dtype=torch.int32)
    slots[:4] = torch.tensor([0, -1, 1, 0])
    p = W.make_projection(1010 + case, T, in_dim, outs, S, r, token_to_slot=slots, with_weight=form == LINEAR)
    d = p.to_device(DEV)
    if form == LINEAR:
        return check_linear(p, d, slots)
    y = d.y.clone()
    LORA.launch_add(y, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=N.IMPL_SGMV)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, slots, 0.5, p.col_offsets), what="scattered rows")
    none = slots < 0
    assert torch.equal(y.cpu()[none].view(torch.int16), p.y[none].view(torch.int16)), "rows without adapter keep their bits"
    if T <= 64:  # one block: a row's result does not depend on where it lies in it
        order = slots.argsort(stable=True)
        z = d.y[order.to(DEV)]
        LORA.launch_add(z, d.x[order.to(DEV)], d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots[order]), 0.5, impl=N.IMPL_SGMV)
        assert torch.equal(z.view(torch.int16), y[order.to(DEV)].view(torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("T, S, impl", [(333, 8, N.IMPL_BGMV), (511, 8, N.IMPL_BGMV), (511, 7, N.IMPL_SGMV), (512, 16, N.IMPL_SGMV), (512, 17, N.IMPL_BGMV)])
def test_few_rows_a_bucket_stay_with_the_bucket_kernel(T, S, impl):
    """Decode batches over few adapters, whose bytes alone would send them to the prefill kernel: 64 rows a bucket below 512 rows, 32 above."""
    slots = torch.arange(T, dtype=torch.int32) * 7 % S
    p = W.make_projection(1040, T, 2048, [6144, 6144], S, 64, token_to_slot=slots)
    d = p.to_device(DEV)
    y = [d.y.clone(), d.y.clone()]
    for out, i in zip(y, (N.IMPL_AUTO, impl)):
        LORA.launch_add(out, d.x, d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, metadata(slots), 0.5, impl=i)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0 and torch.equal(*y)
    assert_lora_close(y[0], O.add_lora(p.y, p.x, p.a_slabs, p.b_slabs, slots, 0.5, p.col_offsets), what="add")
