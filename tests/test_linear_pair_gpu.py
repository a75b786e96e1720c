"""The fused linear of CTA pairs (``csrc/linear_pair.cuh``) at the edges of its 256 x 256 tiles and of its run tables: ragged rows
and columns, runs inside, across and ending at the 128- and 256-row lines, every rank, slices that end inside a tile, and the
form with SiLU * up in the epilogue."""

import pytest
import torch
import torch.nn.functional as F

from helpers import assert_lora_close
from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import workloads as W
from oracle import lora_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def runs(lens, slots, T):
    out = torch.repeat_interleave(torch.tensor(slots, dtype=torch.int32), torch.tensor(lens))
    assert out.numel() == T
    return out


CASES = [
    # T, in, outs, S, r, slots (None: independent rows, a run of almost every row)
    (1536, 64, [4096], 3, 16, runs([128, 128, 300, 84, 896], [0, 1, 2, -1, 0], 1536)),
    (1409, 320, [4096, 224], 4, 64, runs([255, 2, 127, 1, 1024], [3, 0, 1, -1, 2], 1409)),
    (1793, 128, [2080, 32, 1024, 64], 2, 32, runs([1792, 1], [1, 0], 1793)),
    (1300, 192, [4096], 6, 32, None),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_pair_linear_matches_oracle(case):
    T, in_dim, outs, S, r, slots = CASES[case]
    p = W.make_projection(500 + case, T, in_dim, outs, S, r, token_to_slot=slots, with_weight=True)
    d = p.to_device(DEV)
    bias = torch.randn(sum(outs), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    y = LORA.linear_lora(d.x, d.weight, bias.to(DEV), d.a_slabs, d.b_slabs, d.out_sizes, d.col_offsets, d.token_to_slot, 1.0)
    plain = LORA.linear_lora(d.x, d.weight, bias.to(DEV), [], [], [], [], None, 1.0)
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    assert_lora_close(y, O.linear_lora(p.x, p.weight, bias, p.a_slabs, p.b_slabs, p.col_offsets, p.token_to_slot), max_abs=6e-2, what="pair")
    none = p.token_to_slot < 0
    assert torch.equal(y.cpu()[none].view(torch.int16), plain.cpu()[none].view(torch.int16)), "rows without adapter are the plain linear"


@pytest.mark.parametrize("T,in_dim,inter,r,with_lora", [(300, 128, 160, 32, True), (129, 64, 32, 16, False), (1000, 512, 1056, 64, True)])
def test_linear_with_silu_matches_oracle(T, in_dim, inter, r, with_lora):
    S, dev = 3, torch.device(DEV)
    lens = [min(100, T // 2), 1, 27]
    p = W.make_projection(600 + T, T, in_dim, [inter, inter], S, r, with_weight=True,
                          token_to_slot=runs([*lens, T - sum(lens)], [1, -1, 0, 2], T))
    d = p.to_device(DEV)
    y = torch.full((T, inter), 7.0, device=DEV, dtype=torch.bfloat16)
    ws = LORA.scratch_for(dev, N.workspace_bytes(T, 2, r))
    n = 2 if with_lora else 0
    N.check(N.lib().lora_b200_linear_lora_silu(
        y.data_ptr(), inter, d.x.data_ptr(), in_dim, T, in_dim, d.weight.data_ptr(), in_dim, 2 * inter, n, N.ptr_array(d.a_slabs),
        N.ptr_array(d.b_slabs), N.int_array(d.out_sizes), N.int_array(d.col_offsets), S, r, None,
        d.token_to_slot.data_ptr() if n else None, 1.0, ws.data_ptr(), ws.numel(), N.current_stream(dev)))
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    both = p.x.float() @ p.weight.float().T
    if with_lora:
        both = O.add_lora(both, p.x.float(), [a.float() for a in p.a_slabs], [b.float() for b in p.b_slabs], p.token_to_slot, 1.0, p.col_offsets)
    want = F.silu(both[:, :inter].float()) * both[:, inter:].float()
    assert ((y.cpu().float() - want).norm() / want.norm()).item() < 5e-3
