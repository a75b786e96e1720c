"""The kernel for bucketed batches of both 16-bit types (``csrc/bgmv_fused.cuh``): parity with the
CPU oracle at the edges of their tiles - one token, 16- and 32-token chunks and their remainders, partial 128-row output
tiles, K tails and K parts, every rank, popular buckets, mixed ranks, slots of rank 0 - through ``lora_b200_add`` with the
kernel asked for by name."""

import pytest
import torch

from helpers import assert_lora_close
from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import workloads as W
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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("impl", [N.IMPL_BGMV], ids=["bgmv"])
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
