"""The native prefill step (``prefill_layers`` in ``csrc/binding.cpp``) and its attention kernel
(``csrc/prefill_attention.cuh``): attention against an fp32 reference at the edges of its tiles, the step against the
layer-by-layer form of the same decoder."""

import pytest
import torch

from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import backbone as BB
from nanovllm_voxcpm_b200.batch_plan import build_lora_context_from_slot_list
from nanovllm_voxcpm_b200.context import reset_lora_context, set_lora_context

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# q heads, kv heads, head dim, prompt lengths (a CTA covers 16 to 128 positions, a tile 64 keys)
@pytest.mark.parametrize("heads,kv,dim,lens", [
    (16, 2, 64, [1, 63, 64, 65, 15, 16, 17, 200]),
    (8, 2, 128, [129, 1, 127, 128, 31, 33]),
    (3, 3, 64, [130, 5]),
    (12, 2, 128, [70]),
])
def test_prefill_attention_matches_reference(heads, kv, dim, lens):
    gen = torch.Generator(device=DEV).manual_seed(3)
    T = sum(lens)
    ld = (heads + 2 * kv) * dim + 8
    qkv = torch.randn(T, ld, device=DEV, generator=gen).to(torch.bfloat16)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    out = torch.full((T, heads * dim), 9.0, device=DEV, dtype=torch.bfloat16)
    N.check(N.lib().lora_b200_prefill_attention(out.data_ptr(), out.stride(0), qkv.data_ptr(), ld, T, heads, kv, dim, cu.data_ptr(),
                                                len(lens), max(lens), dim ** -0.5, N.current_stream(torch.device(DEV))))
    at = 0
    for n in lens:
        rows = qkv[at:at + n].float()
        q = rows[:, : heads * dim].view(n, heads, dim)
        k = rows[:, heads * dim: (heads + kv) * dim].view(n, kv, dim).repeat_interleave(heads // kv, 1)
        v = rows[:, (heads + kv) * dim: (heads + 2 * kv) * dim].reshape(n, kv, dim).repeat_interleave(heads // kv, 1)
        s = torch.einsum("qhd,khd->hqk", q, k) * dim ** -0.5
        s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        ref = torch.einsum("hqk,khd->qhd", s.softmax(-1), v).reshape(n, heads * dim)
        torch.testing.assert_close(out[at:at + n].float(), ref, rtol=2e-2, atol=2e-2)
        at += n


# rows from below to above the lines between the bucket, prefill and fused-linear kernels; attention by either kernel
@pytest.mark.parametrize("flash", [False, True], ids=["own", "flash"])
@pytest.mark.parametrize("with_lora", [True, False], ids=["lora", "base"])
@pytest.mark.parametrize("dim,lens,r", [(64, [40, 1, 90], 16), (128, [300, 333], 32), (64, [700, 500, 3], 32)])
def test_native_prefill_step_matches_layer_by_layer(dim, lens, r, with_lora, flash, monkeypatch):
    monkeypatch.setattr(BB.Decoder, "_flash_is_faster", lambda *a: flash)
    S, hidden, T = 5, 512, sum(lens)
    cfg = BB.DecoderConfig(hidden_size=hidden, num_heads=8, num_kv_heads=2, head_dim=dim, intermediate_size=768, num_layers=2,
                           max_position=1024, max_loras=S, max_lora_rank=r)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.init_random_(1)
    model.fill_adapter_slots_(S - 1, r, seed=2)
    model.fused_glue = True
    model.allocate_kv_cache(T // cfg.kv_block_size + 1)
    gen = torch.Generator().manual_seed(4)
    embeds = torch.randn(T, hidden, generator=gen).to(DEV, torch.bfloat16)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    step = BB.AttentionStep(True, torch.randperm(T, generator=gen).to(DEV), cu_seqlens=cu, max_seqlen=max(lens))
    positions = torch.cat([torch.arange(n) for n in lens]).to(DEV)
    slots = [s for s, n in zip((1, -1, 3), lens) for _ in range(n)]

    def run(native):
        for layer in model.layers:
            layer.self_attn.k_cache.zero_()
            layer.self_attn.v_cache.zero_()
        prefill, model._prefill_native = model._prefill_native, model._prefill_native if native else lambda *a: None
        try:
            with torch.no_grad():
                if with_lora:
                    set_lora_context(build_lora_context_from_slot_list(slots))
                if native:
                    assert prefill(embeds, positions, step) is not None, "the step was not taken natively"
                out = model(embeds, positions, step)
        finally:
            model._prefill_native = prefill
            reset_lora_context()
        return out, [c.clone() for layer in model.layers for c in (layer.self_attn.k_cache, layer.self_attn.v_cache)]

    got, got_caches = run(True)
    want, want_caches = run(False)
    assert N.device_status(reset=True) == 0
    assert ((got - want).float().norm() / want.float().norm()).item() < 1e-2
    for a, b in zip(got_caches, want_caches):
        assert ((a - b).float().norm() / b.float().norm()).item() < 1e-2


def test_attention_callable_is_checked(monkeypatch):
    cfg = BB.DecoderConfig(hidden_size=128, num_heads=2, num_kv_heads=1, head_dim=64, intermediate_size=128, num_layers=1, max_position=64,
                           max_loras=2, max_lora_rank=16)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.allocate_kv_cache(1)
    reset_lora_context()
    step = BB.AttentionStep(True, torch.arange(4, device=DEV), cu_seqlens=torch.tensor([0, 4], dtype=torch.int32, device=DEV), max_seqlen=4)
    embeds, positions = torch.zeros(4, 128, device=DEV, dtype=torch.bfloat16), torch.arange(4, device=DEV)
    monkeypatch.setattr(BB.Decoder, "_flash_is_faster", lambda *a: True)
    for bad in (lambda qkv: qkv, lambda qkv: qkv[:, :128], lambda qkv: None, lambda qkv: qkv[:, :128].float().contiguous()):
        monkeypatch.setattr(BB.Decoder, "_flash_attend", lambda self, s, bad=bad: bad)
        with pytest.raises(TypeError, match="attend"):
            model._prefill_native(embeds, positions, step)

    def fails(qkv):
        raise KeyError("out of blocks")

    monkeypatch.setattr(BB.Decoder, "_flash_attend", lambda self, s: fails)
    with pytest.raises(KeyError, match="out of blocks"):
        model._prefill_native(embeds, positions, step)


@pytest.mark.parametrize("lens,fused", [([4] * 32, False), ([47] * 3, False), ([48] * 3, True), ([200, 56], True)])
def test_projections_of_short_prompts_are_not_fused(lens, fused):
    """1024 input columns, rank 32: fewer than 48 rows a prompt go to cuBLAS and the add, as layer by layer (the same bits of v in the
    first layer's cache); the fused linear, which rounds the sum once, takes the others."""
    T, S = sum(lens), 6
    cfg = BB.DecoderConfig(hidden_size=1024, num_heads=8, num_kv_heads=2, head_dim=64, intermediate_size=256, num_layers=1, max_position=256,
                           max_loras=S, max_lora_rank=32)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.init_random_(1)
    model.fill_adapter_slots_(S, 32, seed=2)
    model.fused_glue = True
    model.allocate_kv_cache(T // cfg.kv_block_size + 1)
    embeds = torch.randn(T, 1024, generator=torch.Generator().manual_seed(4)).to(DEV, torch.bfloat16)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    step = BB.AttentionStep(True, torch.arange(T, device=DEV), cu_seqlens=cu, max_seqlen=max(lens))
    positions = torch.cat([torch.arange(n) for n in lens]).to(DEV)
    native, caches = model._prefill_native, []
    for take in (native, lambda *a: None):
        model._prefill_native = take
        try:
            with torch.no_grad():
                set_lora_context(build_lora_context_from_slot_list([i % S for i, n in enumerate(lens) for _ in range(n)]))
                model(embeds, positions, step)
        finally:
            reset_lora_context()
        caches.append(model.layers[0].self_attn.v_cache.clone())
    assert N.device_status(reset=True) == 0
    torch.testing.assert_close(caches[0], caches[1], rtol=1e-2, atol=2e-2)
    assert torch.equal(*caches) != fused
