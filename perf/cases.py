"""Performance cases of the package: the calls that a serving process makes through the public entry points.

Kinds of case
  decode      multi-LoRA adds of a decode batch (one row per sequence) over the four projections of `layers` decoder
              layers, each with slabs of its own; issued eagerly or replayed from a CUDA graph whose index buffers
              hold one bucket per resident adapter
  prefill     the same calls for a batch of whole prompts (rows of a request contiguous, one adapter per request)
  linear      base GEMM and multi-LoRA delta in one call (``linear_lora``) for a batch of whole prompts
  ops         ``lora_shrink`` then ``lora_expand`` with the vLLM-style metadata, as an operator-level caller has them
  dec_decode  a decode step of a decoder: index build on the device, then the replayed graph of all layers
  dec_prefill an eager prefill step of a decoder: batch plan built from the step's slot list, then all layers
  admission   one adapter checkpoint, read into pinned host memory, loaded into a resident slot of every module

Widths are those of this repository's configurations: hidden 1024 with 16 / 2 heads of 64 and intermediate 4096, hidden
2048 with 16 / 2 heads of 128 and intermediate 6144, hidden 4096 with 32 / 8 heads of 128 and intermediate 14336; `tp` is
the number of tensor-parallel ranks whose per-rank shapes are used.
"""

from __future__ import annotations

import math
import os
import tempfile

import torch

from nanovllm_voxcpm_b200 import adapter_checkpoint as AC
from nanovllm_voxcpm_b200 import backbone as BB
from nanovllm_voxcpm_b200 import layers as L
from nanovllm_voxcpm_b200 import lora as LORA
from nanovllm_voxcpm_b200 import lora_ops as OPS
from nanovllm_voxcpm_b200.batch_plan import (
    GraphLoRABuffers,
    build_lora_batch_plan_from_token_to_slot,
    build_lora_context_from_batch_plan,
    build_lora_context_from_slot_list,
)
from nanovllm_voxcpm_b200.context import set_lora_context
from nanovllm_voxcpm_b200.slot_loader import SlotLoader

#: hidden size -> (query heads, kv heads, head dim, intermediate size)
FAMILIES = {1024: (16, 2, 64, 4096), 2048: (16, 2, 128, 6144), 4096: (32, 8, 128, 14336)}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one user, one token: nothing but latency, the call overhead of an eager engine included
        dict(name="decode_1row_eager", kind="decode", T=1, S=8, none=0.0, spread="uniform", hidden=1024, tp=1, r=32,
             mixed=False, dtype="bf16", graph=False, layers=2),
        # a full decode batch over 32 adapters (the decode configuration), replayed as engines do
        dict(name="decode_256rows_graph", kind="decode", T=256, S=32, none=0.1, spread="uniform", hidden=1024, tp=1, r=32,
             mixed=False, dtype="bf16", graph=True, layers=4),
        # a half-empty batch with small adapters (rank 16 is the rank of the smallest configuration)
        dict(name="decode_37rows_rank16", kind="decode", T=37, S=16, none=0.25, spread="uniform", hidden=1024, tp=1, r=16,
             mixed=False, dtype="bf16", graph=True, layers=4),
        # the largest decode batch: wide layers, rank 64, hundreds of resident adapters with a skewed popularity
        dict(name="decode_512rows_wide", kind="decode", T=512, S=176, none=0.0, spread="zipf", hidden=4096, tp=1, r=64,
             mixed=False, dtype="bf16", graph=True, layers=1),
        # a model kept in half precision, eager, adapters of different ranks in one slab
        dict(name="decode_64rows_fp16", kind="decode", T=64, S=32, none=0.1, spread="zipf", hidden=1024, tp=1, r=32,
             mixed=True, dtype="fp16", graph=False, layers=2),
        # a full prefill batch (the prefill configuration): 16 ragged prompts, ranks 8 / 16 / 64 in a rank-64 slab
        dict(name="prefill_8172rows", kind="prefill", T=8172, reqs=16, S=16, none=0.0, hidden=2048, tp=1, r=64, mixed=True,
             dtype="bf16"),
        # three short prompts: the usual prefill of a lightly loaded server
        dict(name="prefill_301rows", kind="prefill", T=301, reqs=3, S=32, none=0.0, hidden=1024, tp=1, r=32, mixed=False,
             dtype="bf16"),
        # the fused linear on the prefill configuration: the largest arithmetic of a step
        dict(name="linear_8172rows", kind="linear", T=8172, reqs=16, S=16, none=0.0, hidden=2048, tp=1, r=64, mixed=True,
             dtype="bf16"),
        # operator-level callers: shrink and expand as two calls around an intermediate of their own
        dict(name="ops_200rows", kind="ops", T=200, S=32, none=0.1, spread="uniform", hidden=1024, tp=1, r=32, mixed=False,
             dtype="bf16"),
        # a decode step of 64 concurrent requests with 128 resident adapters
        dict(name="dec_decode_64reqs", kind="dec_decode", T=64, S=128, none=0.0, hidden=1024, r=32, layers=8, ctx=352),
        # the prefill step that admits a dozen of those requests
        dict(name="dec_prefill_4001rows", kind="dec_prefill", T=4001, reqs=12, S=128, none=0.0, hidden=1024, r=32, layers=4),
        # an adapter comes in while the server runs
        dict(name="admission_rank32", kind="admission", S=8, hidden=2048, r=32, rank=32, layers=4),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choices(["decode", "prefill", "linear", "ops", "dec_decode", "dec_prefill", "admission"],
                       [40, 22, 8, 8, 9, 6, 7])[0]
    if kind == "decode":
        hidden = rng.choice([1024, 1024, 2048, 4096])
        r = rng.choice([16, 32, 32, 64])
        S = _log_int(rng, 4, 128 if hidden < 4096 else 96)
        return dict(kind=kind, T=_log_int(rng, 1, 384), S=S, none=rng.choice([0.0, 0.1, 0.25]),
                    spread=rng.choice(["uniform", "zipf"]), hidden=hidden, tp=rng.choice([1, 1, 2, 4]) if hidden == 4096 else 1,
                    r=r, mixed=rng.random() < 0.3, dtype="fp16" if rng.random() < 0.15 else "bf16", graph=rng.random() < 0.6,
                    layers=1 if hidden == 4096 else rng.choice([2, 3, 4]))
    if kind in ("prefill", "linear"):
        hidden = rng.choice([1024, 2048, 2048])
        T = _log_int(rng, 64, 8000)
        return dict(kind=kind, T=T, reqs=min(max(1, T // 40), _log_int(rng, 1, 16)), S=_log_int(rng, 4, 32),
                    none=rng.choice([0.0, 0.0, 0.2]), hidden=hidden, tp=1, r=rng.choice([16, 32, 64]), mixed=rng.random() < 0.4,
                    dtype="fp16" if kind == "prefill" and rng.random() < 0.15 else "bf16")
    if kind == "ops":
        return dict(kind=kind, T=_log_int(rng, 8, 3000), S=_log_int(rng, 4, 64), none=rng.choice([0.0, 0.1, 0.25]),
                    spread=rng.choice(["uniform", "zipf"]), hidden=rng.choice([1024, 2048]), tp=1, r=rng.choice([16, 32, 64]),
                    mixed=False, dtype="bf16")
    if kind == "dec_decode":
        return dict(kind=kind, T=_log_int(rng, 1, 128), S=_log_int(rng, 8, 128), none=rng.choice([0.0, 0.1]),
                    hidden=rng.choice([1024, 1024, 2048]), r=rng.choice([16, 32]), layers=rng.choice([2, 4, 6]),
                    ctx=_log_int(rng, 64, 640))
    if kind == "dec_prefill":
        T = _log_int(rng, 128, 4000)
        return dict(kind=kind, T=T, reqs=min(max(1, T // 60), _log_int(rng, 1, 12)), S=_log_int(rng, 8, 128),
                    none=rng.choice([0.0, 0.1]), hidden=rng.choice([1024, 1024, 2048]), r=rng.choice([16, 32]),
                    layers=rng.choice([2, 3, 4]))
    r = rng.choice([16, 32, 64])
    return dict(kind=kind, S=8, hidden=rng.choice([1024, 2048]), r=r, rank=rng.choice([q for q in (8, 16, 32, 64) if q <= r]),
                layers=rng.choice([1, 2, 3, 4]))


# --------------------------------------------------------------------------------------------- shapes and routing
def _projections(case):
    """(input width, slice widths) of the four projections of a decoder layer on one tensor-parallel rank."""
    heads, kv, dim, inter = FAMILIES[case["hidden"]]
    tp = case.get("tp", 1)
    q, k, i = heads * dim // tp, kv * dim // tp, inter // tp
    return [(case["hidden"], [q, k, k]), (q, [case["hidden"]]), (case["hidden"], [i, i]), (i, [case["hidden"]])]


def _ranks(case):
    return [(8, 16, case["r"])[s % 3] if case.get("mixed") else case["r"] for s in range(case["S"])]


def _popularity(case):
    S = case["S"]
    if case.get("spread", "zipf") == "uniform":
        return torch.full((S,), 1.0 / S, dtype=torch.float64)
    w = 1.0 / torch.arange(1, S + 1, dtype=torch.float64) ** 1.1
    return w / w.sum()


def _lengths(case, gen):
    """Ragged prompt lengths that sum to T (each at least a quarter of the mean)."""
    n, T = case["reqs"], case["T"]
    w = torch.rand(n, generator=gen, dtype=torch.float64) + 0.15
    lens = [max(1, int(v)) for v in (w / w.sum() * T)]
    lens[0] += T - sum(lens)
    return lens


def _slots(case, seed):
    """Slot of every row: independent rows in decode, one slot per request in prefill; `none` of them without adapter."""
    gen = torch.Generator().manual_seed(1000 + seed)
    n = case.get("reqs", case["T"])
    slots = torch.multinomial(_popularity(case), n, replacement=True, generator=gen)
    drop = torch.rand(n, generator=gen) < case["none"]
    drop[0] = False  # a batch without any adapter makes no multi-LoRA call
    slots[drop] = -1
    if "reqs" not in case:
        return slots.tolist(), [1] * n
    lens = _lengths(case, gen)
    return [int(s) for s, m in zip(slots, lens) for _ in range(m)], lens


def _metadata(ctx):
    return LORA.LoRAMetadata(ctx.token_to_slot, ctx.token_indices_sorted_by_slot, ctx.active_slot_ids,
                             ctx.num_tokens_per_slot, ctx.slot_start_offsets, ctx.no_lora_flag, ctx.num_active_loras)


def _adapters(case, in_dim, outs, gen, dtype):
    """Slabs [S, r, in] and [S, out, r] of one projection, zero beyond each slot's rank."""
    S, r = case["S"], case["r"]
    rank = torch.tensor(_ranks(case), device="cuda")
    live = torch.arange(r, device="cuda")[None, :] < rank[:, None]
    draw_ = lambda *shape: torch.empty(*shape, device="cuda", dtype=dtype).normal_(0.0, 0.02, generator=gen)  # noqa: E731
    a = [draw_(S, r, in_dim) * live[:, :, None] for _ in outs]
    b = [draw_(S, out, r) * live[:, None, :] for out in outs]
    return a, b


def _calls(case, gen, dtype):
    """One multi-LoRA call per projection and layer: x, the base output y that it updates, and the layer's slabs."""
    calls, T = [], case["T"]
    rn = lambda *shape: torch.empty(*shape, device="cuda", dtype=dtype).normal_(generator=gen)  # noqa: E731
    ranks = torch.tensor(_ranks(case), dtype=torch.int32, device="cuda")
    for _ in range(case.get("layers", 1)):
        for in_dim, outs in _projections(case):
            a, b = _adapters(case, in_dim, outs, gen, dtype)
            y = rn(T, sum(outs))
            calls.append(dict(x=rn(T, in_dim), y=y, views=list(y.split(outs, dim=-1)), a=a, b=b, outs=outs,
                              cols=[sum(outs[:i]) for i in range(len(outs))], ranks=ranks))
    return calls


def _adds(state):
    backend, meta = state["backend"], state["meta"]
    for c in state["calls"]:
        backend.add_lora(c["views"], c["x"], c["a"], c["b"], indices=meta.token_to_slot, metadata=meta, scaling=1.0,
                         y_packed=c["y"], rank_per_slot=c["ranks"])


def _capture(fn):
    """CUDA graph of `fn` after two ordinary runs on a side stream, as an engine captures its decode step."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fn()
        fn()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        fn()
    torch.cuda.synchronize()
    return graph


# --------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    with torch.inference_mode():
        state = globals()["_prepare_" + case["kind"]](case, seed, torch.Generator(device="cuda").manual_seed(seed))
    state["kind"] = case["kind"]
    return state


def _prepare_decode(case, seed, gen):
    slots, _ = _slots(case, seed)
    state = dict(backend=LORA.get_backend(), calls=_calls(case, gen, DTYPES[case["dtype"]]), graph=None)
    if not case["graph"]:
        state["meta"] = _metadata(build_lora_context_from_slot_list(slots))
        return state
    state["buffers"] = GraphLoRABuffers.make(case["T"], case["S"])
    state["buffers"].load_plan(build_lora_batch_plan_from_token_to_slot({}, slots))
    state["meta"] = _metadata(state["buffers"].context(case["T"]))
    fresh = [c["y"].clone() for c in state["calls"]]
    state["graph"] = _capture(lambda: _adds(state))
    for c, y in zip(state["calls"], fresh):
        c["y"].copy_(y)
    return state


def _prepare_prefill(case, seed, gen):
    slots, _ = _slots(case, seed)
    return dict(backend=LORA.get_backend(), calls=_calls(case, gen, DTYPES[case["dtype"]]), graph=None,
                meta=_metadata(build_lora_context_from_slot_list(slots)))


def _prepare_linear(case, seed, gen):
    state = _prepare_prefill(case, seed, gen)
    for c in state["calls"]:
        in_dim = c["x"].size(1)
        c["w"] = torch.empty(sum(c["outs"]), in_dim, device="cuda", dtype=c["x"].dtype).normal_(0.0, 0.02, generator=gen)
    return state


def _prepare_ops(case, seed, gen):
    slots, _ = _slots(case, seed)
    meta = OPS.LoRAKernelMeta.make(case["S"], case["T"], "cuda")
    meta.prepare_tensors(torch.tensor(slots, dtype=torch.int32, device="cuda"))
    calls = _calls(case, gen, DTYPES[case["dtype"]])
    for c in calls:
        c["tmp"] = torch.zeros(len(c["outs"]), case["T"], case["r"], device="cuda", dtype=c["x"].dtype)
    return dict(calls=calls, args=meta.meta_args(case["T"], specialize_active_lora=True))


def _decoder(case, seed, max_position):
    heads, kv, dim, inter = FAMILIES[case["hidden"]]
    cfg = BB.DecoderConfig(hidden_size=case["hidden"], num_heads=heads, num_kv_heads=kv, head_dim=dim, intermediate_size=inter,
                           num_layers=case["layers"], max_position=max_position, max_loras=case["S"], max_lora_rank=case["r"])
    with torch.device("cuda"):
        model = BB.Decoder(cfg).to(torch.bfloat16)
    model.fused_glue = True
    return model, cfg


def _prepare_dec_decode(case, seed, gen):
    T, ctx = case["T"], case["ctx"]
    model, cfg = _decoder(case, seed, 1024)
    model.init_random_(seed)
    model.fill_adapter_slots_(case["S"], case["r"], seed=seed + 1)
    # requests at positions around `ctx`, each with its own blocks of the paged cache
    lens = torch.randint(max(1, ctx // 2), ctx + ctx // 2, (T,), generator=torch.Generator().manual_seed(seed)).cuda()
    per = -(-(ctx + ctx // 2 + 1) // cfg.kv_block_size)
    model.allocate_kv_cache(T * per)
    for layer in model.layers:
        layer.self_attn.k_cache.normal_(generator=gen)
        layer.self_attn.v_cache.normal_(generator=gen)
    blocks = torch.arange(T * per, dtype=torch.int32, device="cuda").view(T, per)
    at = blocks[torch.arange(T, device="cuda"), lens // cfg.kv_block_size].long() * cfg.kv_block_size + lens % cfg.kv_block_size
    step = BB.AttentionStep(False, at, context_lens=(lens + 1).to(torch.int32), block_tables=blocks)
    embeds = torch.empty(T, case["hidden"], device="cuda", dtype=torch.bfloat16).normal_(generator=gen)
    buffers = GraphLoRABuffers.make(T, case["S"])
    slots = torch.tensor(_slots(case, seed)[0], dtype=torch.int32, device="cuda")
    buffers.load_token_to_slot_on_device(slots)
    out = torch.empty_like(embeds)

    def forward():
        set_lora_context(buffers.context(T))
        out.copy_(model(embeds, lens, step))

    return dict(model=model, buffers=buffers, slots=slots, out=out, keep=(embeds, lens, step), graph=_capture(forward))


def _prepare_dec_prefill(case, seed, gen):
    slots, lens = _slots(case, seed)
    model, cfg = _decoder(case, seed, 8192)
    model.init_random_(seed)
    model.fill_adapter_slots_(case["S"], case["r"], seed=seed + 1)
    blocks = [-(-n // cfg.kv_block_size) for n in lens]
    model.allocate_kv_cache(case["T"] // cfg.kv_block_size + len(lens))
    first = [sum(blocks[:i]) * cfg.kv_block_size for i in range(len(lens))]
    at = torch.cat([f + torch.arange(n) for f, n in zip(first, lens)]).cuda()
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    positions = torch.cat([torch.arange(n) for n in lens]).cuda()
    embeds = torch.empty(case["T"], case["hidden"], device="cuda", dtype=torch.bfloat16).normal_(generator=gen)
    return dict(model=model, slots=slots, embeds=embeds, positions=positions,
                step=BB.AttentionStep(True, at, cu_seqlens=cu, max_seqlen=max(lens)))


def _prepare_admission(case, seed, gen):
    model, cfg = _decoder(case, seed, 64)
    modules = {n: m for n, m in model.named_modules() if isinstance(m, L._LORA_LAYER_TYPES)}
    unpack = {"qkv_proj": ("q_proj", "k_proj", "v_proj"), "gate_up_proj": ("gate_proj", "up_proj")}
    tensors = {}
    rn = lambda *shape: torch.empty(*shape, device="cuda").normal_(0.0, 0.02, generator=gen).cpu()  # noqa: E731
    for name, m in modules.items():
        parent, _, leaf = name.rpartition(".")
        for proj, a, b in zip(unpack.get(leaf, (leaf,)), m._a_slices(), m._b_slices()):
            tensors[f"{parent}.{proj}.lora_A"] = rn(case["rank"], a.size(2))
            tensors[f"{parent}.{proj}.lora_B"] = rn(b.size(1), case["rank"])
    with tempfile.TemporaryDirectory() as root:
        path = AC.save_lora_checkpoint(os.path.join(root, "adapter"), tensors, rank=case["rank"], alpha=2.0 * case["rank"])
        payload = AC.load_lora_checkpoint(str(path))
    return dict(model=model, loader=SlotLoader(model), payload=payload, slot=0, n_slots=case["S"], modules=list(modules.values()))


# --------------------------------------------------------------------------------------------- run
def run(state):
    with torch.inference_mode():
        return globals()["_run_" + state["kind"]](state)


def _run_decode(state):
    if state["graph"] is not None:
        state["graph"].replay()
    else:
        _adds(state)
    return [c["y"] for c in state["calls"]]


_run_prefill = _run_decode


def _run_linear(state):
    return [LORA.linear_lora(c["x"], c["w"], None, c["a"], c["b"], c["outs"], c["cols"], state["meta"].token_to_slot, 1.0)
            for c in state["calls"]]


def _run_ops(state):
    for c in state["calls"]:
        OPS.lora_shrink(c["x"], c["a"], c["tmp"], *state["args"], 1.0)
        OPS.lora_expand(c["tmp"], c["b"], c["y"], *state["args"], offset_start=0, add_inputs=True)
    return [t for c in state["calls"] for t in (c["tmp"], c["y"])]


def _caches(model):
    return [c for layer in model.layers for c in (layer.self_attn.k_cache, layer.self_attn.v_cache)]


def _run_dec_decode(state):
    state["buffers"].load_token_to_slot_on_device(state["slots"])
    state["graph"].replay()
    return [state["out"], *_caches(state["model"])]


def _run_dec_prefill(state):
    plan = build_lora_batch_plan_from_token_to_slot({}, state["slots"])
    set_lora_context(build_lora_context_from_batch_plan(plan))
    return [state["model"](state["embeds"], state["positions"], state["step"]), *_caches(state["model"])]


def _run_admission(state):
    slot = state["slot"]
    state["slot"] = (slot + 1) % state["n_slots"]
    state["loader"].load_slot(slot, state["payload"])
    return [slab[slot] for m in state["modules"] for slab in (*m._a_slices(), *m._b_slices())]


# --------------------------------------------------------------------------------------------- work and tolerance
def _lora_work(case):
    """Bytes and operations of the adapter part of one layer: weights of the adapters in use (at their ranks) once, rows
    with an adapter of x once, of y read and written."""
    slots = [s for s in _slots(case, 0)[0] if s >= 0]
    ranks = _ranks(case)
    nbytes = flops = 0
    for in_dim, outs in _projections(case):
        per_rank = len(outs) * in_dim + sum(outs)
        nbytes += 2 * sum(ranks[s] for s in set(slots)) * per_rank
        nbytes += 2 * len(slots) * (in_dim + 2 * sum(outs))
        flops += 2 * sum(ranks[s] for s in slots) * per_rank
    return nbytes, flops


def work(case):
    kind, T = case["kind"], case.get("T", 0)
    if kind == "admission":
        per_rank = sum(len(outs) * in_dim + sum(outs) for in_dim, outs in _projections(case))
        n = case["layers"] * per_rank
        return {"bytes": 4 * n * case["rank"] + 2 * n * case["r"], "flops": n * case["rank"]}
    nbytes, flops = _lora_work(case)
    weights = sum(in_dim * sum(outs) for in_dim, outs in _projections(case))
    io = sum(in_dim + sum(outs) for in_dim, outs in _projections(case))
    if kind == "linear":
        with_adapter = sum(s >= 0 for s in _slots(case, 0)[0])
        nbytes += 2 * weights + 2 * T * io - 2 * with_adapter * sum(in_dim + 2 * sum(outs) for in_dim, outs in _projections(case))
        flops += 2 * T * weights
    elif kind == "ops":
        nbytes += 2 * T * case["r"] * sum(len(outs) for _, outs in _projections(case)) * 2
    elif kind in ("dec_decode", "dec_prefill"):
        # adapters and base weights once a layer; the hidden rows stay on the chip at best, the caches are read / written
        heads, kv, dim, _ = FAMILIES[case["hidden"]]
        slots = [s for s in _slots(case, 0)[0] if s >= 0]
        adapters = 2 * case["r"] * len(set(slots)) * sum(len(outs) * in_dim + sum(outs) for in_dim, outs in _projections(case))
        cached = 2 * 2 * T * kv * dim
        pairs = T * case["ctx"] if kind == "dec_decode" else sum(n * n / 2 for n in _slots(case, 0)[1])
        if kind == "dec_decode":
            cached += 2 * 2 * T * case["ctx"] * kv * dim
        nbytes = case["layers"] * (adapters + 2 * weights + cached) + 2 * 2 * T * case["hidden"]
        flops = case["layers"] * (flops + 2 * T * weights + 4 * pairs * heads * dim)
    elif kind == "decode":
        nbytes, flops = case["layers"] * nbytes, case["layers"] * flops
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "admission":
        return "exact"
    if case["kind"].startswith("dec_"):
        return {"rel": 2e-2}  # bf16 roundings of a stack of layers
    return {"rel": 1e-2 if case.get("dtype") != "fp16" else 2e-3}
