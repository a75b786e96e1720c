"""The short decode chain (``csrc/decode_step.cuh``) against the layer-by-layer step of the same decoder (library GEMMs, LoRA add,
flash_attn, separate glue kernels): outputs within the rounding of a bf16 stack, the new rows of the caches equal up to the
projection's rounding, rows without adapter as in the decoder without adapters, graph replay equal to eager launches."""

import pytest
import torch

from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import backbone as BB
from nanovllm_voxcpm_b200.batch_plan import GraphLoRABuffers
from nanovllm_voxcpm_b200.context import reset_lora_context, set_lora_context

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# rows, q heads, kv heads, head dim, hidden, intermediate, rank, longest context (a warp takes blocks of 16 tokens, eight warps in turn)
CASES = [
    (1, 16, 2, 64, 1024, 4096, 32, 40),
    (17, 16, 2, 64, 1024, 4096, 16, 800),
    (37, 8, 2, 128, 512, 320, 64, 430),
    (128, 4, 4, 64, 256, 192, 32, 17),
]


@pytest.mark.parametrize("with_lora", [True, False], ids=["lora", "base"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_chain_matches_the_layer_by_layer_step(case, with_lora):
    T, heads, kv, dim, hidden, inter, r, longest = CASES[case]
    S = 6
    cfg = BB.DecoderConfig(hidden_size=hidden, num_heads=heads, num_kv_heads=kv, head_dim=dim, intermediate_size=inter, num_layers=2,
                           max_position=1024, max_loras=S, max_lora_rank=r)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.init_random_(case)
    model.fill_adapter_slots_(S - 1, r, seed=case + 1)  # the last slot stays empty (rank 0)
    model.fused_glue = True
    gen = torch.Generator().manual_seed(case)
    lens = torch.randint(0, longest, (T,), generator=gen)
    lens[0] = longest - 1
    per = -(-longest // cfg.kv_block_size)
    tables = torch.randperm(T * per, generator=gen).to(torch.int32).view(T, per).to(DEV)
    lens = lens.to(DEV)
    at = tables[torch.arange(T, device=DEV), lens // cfg.kv_block_size].long() * cfg.kv_block_size + lens % cfg.kv_block_size
    step = BB.AttentionStep(False, at, context_lens=(lens + 1).to(torch.int32), block_tables=tables)
    embeds = torch.randn(T, hidden, generator=gen).to(DEV, torch.bfloat16)
    slots = torch.randint(-1, S, (T,), generator=gen, dtype=torch.int32)
    model.allocate_kv_cache(T * per)
    filled = [torch.randn(model.layers[0].self_attn.k_cache.shape, generator=gen).to(DEV, torch.bfloat16) for _ in range(4)]

    def caches():
        return [c for layer in model.layers for c in (layer.self_attn.k_cache, layer.self_attn.v_cache)]

    def run(chain, lora, graph=False):
        for c, f in zip(caches(), filled):
            c.copy_(f)
        ok = type(model)._decode_chain_ok
        if lora:
            bufs = GraphLoRABuffers.make(T, S, device=DEV)
            bufs.load_token_to_slot_on_device(slots.to(DEV))
            set_lora_context(bufs.context(T))
        else:
            reset_lora_context()
        try:
            if not chain:
                type(model)._decode_chain_ok = lambda *a: False
            else:
                assert model._decode_chain_ok(embeds, lens, step)
            with torch.inference_mode():
                if not graph:
                    out = model(embeds, lens, step)
                else:
                    stream = torch.cuda.Stream()
                    with torch.cuda.stream(stream):
                        model(embeds, lens, step)
                    stream.synchronize()
                    g = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g, stream=stream):
                        out = model(embeds, lens, step)
                    g.replay()
                torch.cuda.synchronize()
        finally:
            type(model)._decode_chain_ok = ok
            reset_lora_context()
        return out.float().clone(), [c.float().clone() for c in caches()]

    out, kv_new = run(True, with_lora)
    ref, kv_ref = run(False, with_lora)
    torch.testing.assert_close(out, ref, atol=4e-2, rtol=4e-2)
    for a, b in zip(kv_new, kv_ref):
        torch.testing.assert_close(a, b, atol=4e-2, rtol=4e-2)
    flat = kv_new[0].view(-1, kv, dim)
    keep = torch.ones(flat.size(0), dtype=torch.bool, device=DEV)
    keep[at] = False
    assert torch.equal(flat[keep], filled[0].float().view(-1, kv, dim)[keep]), "rows of the cache that are not new changed"
    again, _ = run(True, with_lora, graph=True)
    assert torch.equal(again, out)
    if with_lora:
        base, _ = run(True, False)
        none = ((slots < 0) | (slots == S - 1)).to(DEV)
        assert torch.equal(out[none], base[none]), "rows without adapter differ from the decoder without adapters"
        assert T == 1 or not torch.equal(out[~none], base[~none])
    assert N.device_status(reset=True) == 0


def test_step_at_a_rank_that_the_chain_does_not_take():
    """Rank 176 in three slices is more than a cluster holds: the step runs layer by layer."""
    T, S, hidden = 5, 3, 256
    cfg = BB.DecoderConfig(hidden_size=hidden, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=128, num_layers=2,
                           max_position=64, max_loras=S, max_lora_rank=176)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.init_random_(0)
    model.fill_adapter_slots_(S, 176, seed=1)
    model.allocate_kv_cache(T)
    lens = torch.arange(3, 3 + T, device=DEV)
    tables = torch.arange(T, dtype=torch.int32, device=DEV).view(T, 1)
    step = BB.AttentionStep(False, tables[:, 0].long() * cfg.kv_block_size + lens, context_lens=(lens + 1).to(torch.int32), block_tables=tables)
    embeds = torch.randn(T, hidden, generator=torch.Generator().manual_seed(0)).to(DEV, torch.bfloat16)
    bufs = GraphLoRABuffers.make(T, S, device=DEV)
    bufs.load_token_to_slot_on_device(torch.tensor([0, 1, -1, 2, 0], dtype=torch.int32, device=DEV))
    set_lora_context(bufs.context(T))
    try:
        with torch.inference_mode():
            model.fused_glue = True
            assert not model._decode_chain_ok(embeds, lens, step)
            got = model(embeds, lens, step)
            model.fused_glue = False
            want = model(embeds, lens, step)
    finally:
        reset_lora_context()
    torch.testing.assert_close(got.float(), want.float(), atol=4e-2, rtol=4e-2)
    assert N.device_status(reset=True) == 0


def _strided(t):
    """The same values with a gap behind each."""
    wide = torch.zeros(*t.shape, 2, dtype=t.dtype, device=t.device)
    wide[..., 0] = t
    return wide[..., 0]


@pytest.mark.parametrize("what", ["positions", "slot_mapping", "context_lens", "block_tables", "k_cache", "block size", "norm", "token_to_slot",
                                  "counts", "embeds"])
def test_forms_that_the_chain_would_misread_run_layer_by_layer(what):
    T, S, hidden = 5, 3, 256
    cfg = BB.DecoderConfig(hidden_size=hidden, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=128, num_layers=1,
                           max_position=64, max_loras=S, max_lora_rank=16)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.fused_glue = True
    model.allocate_kv_cache(2 * T)
    lens = torch.arange(3, 3 + T, device=DEV)
    tables = torch.arange(2 * T, dtype=torch.int32, device=DEV).view(T, 2)
    step = BB.AttentionStep(False, tables[:, 0].long() * cfg.kv_block_size + lens, context_lens=(lens + 1).to(torch.int32), block_tables=tables)
    embeds = torch.randn(T, hidden, device=DEV, dtype=torch.bfloat16)
    bufs = GraphLoRABuffers.make(T, S, device=DEV)
    bufs.load_token_to_slot_on_device(torch.tensor([0, 1, -1, 2, 0], dtype=torch.int32, device=DEV))
    ctx = bufs.context(T)
    set_lora_context(ctx)
    try:
        assert model._decode_chain_ok(embeds, lens, step)
        sa = model.layers[0].self_attn
        if what == "positions":
            lens = _strided(lens)
        elif what in ("slot_mapping", "context_lens", "block_tables"):
            setattr(step, what, _strided(getattr(step, what)))
        elif what == "k_cache":
            sa.k_cache = _strided(sa.k_cache)
        elif what == "block size":
            sa.k_cache = sa.k_cache.view(-1, cfg.kv_block_size * 2, 2, 64)
        elif what == "norm":
            model.norm.data = model.norm.data.float()
        elif what == "token_to_slot":
            ctx.token_to_slot = _strided(ctx.token_to_slot)
        elif what == "counts":
            ctx.num_tokens_per_slot = ctx.num_tokens_per_slot.long()
        else:
            embeds = _strided(embeds)
        assert not model._decode_chain_ok(embeds, lens, step)
    finally:
        reset_lora_context()


def test_strided_slot_mapping_gives_the_same_step():
    """A form that the layer-by-layer step takes (it converts the map)."""
    T, hidden = 5, 256
    cfg = BB.DecoderConfig(hidden_size=hidden, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=128, num_layers=1,
                           max_position=64, max_loras=2, max_lora_rank=16)
    with torch.device(DEV):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.fused_glue = True
    model.init_random_(0)
    lens = torch.arange(3, 3 + T, device=DEV)
    tables = torch.arange(T, dtype=torch.int32, device=DEV).view(T, 1)
    at = tables[:, 0].long() * cfg.kv_block_size + lens
    embeds = torch.randn(T, hidden, device=DEV, dtype=torch.bfloat16)
    out = []
    for slots in (at, _strided(at)):
        model.allocate_kv_cache(T)
        step = BB.AttentionStep(False, slots, context_lens=(lens + 1).to(torch.int32), block_tables=tables)
        with torch.inference_mode():
            out.append((model(embeds, lens, step).float(), model.layers[0].self_attn.k_cache.float()))
    torch.testing.assert_close(out[1][0], out[0][0], atol=4e-2, rtol=4e-2)
    torch.testing.assert_close(out[1][1], out[0][1], atol=4e-2, rtol=4e-2)
