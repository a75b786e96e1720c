"""The two kernels of the decode chain that compute something (``csrc/decode_step.cuh``) against 64-bit references: the projection
with its fp32 planes (base product and LoRA delta), and attention over planes and the paged cache with RoPE and the cache store."""

import pytest
import torch

from nanovllm_voxcpm_b200 import _native as N
from test_parity_gpu import metadata_for

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# rows, in, slices, rank; 128-row weight tiles, 64-column K steps and 1 to 8 K parts, windows of 16 rows, both kinds of delta
LINEAR = [
    (1, 64, [8], 16),
    (16, 1024, [1024, 128, 128], 32),
    (17, 192, [136, 40], 48),
    (37, 4096, [1024], 32),
    (64, 1024, [4096, 4096], 64),
    (100, 2048, [2048, 256, 256], 160),
    (127, 6144, [2048], 64),
    (128, 320, [520], 256),
]


@pytest.mark.parametrize("with_lora", [True, False], ids=["lora", "base"])
@pytest.mark.parametrize("case", range(len(LINEAR)))
def test_decode_linear_planes(case, with_lora):
    T, in_dim, outs, r = LINEAR[case]
    S, out = 5, sum(outs)
    gen = torch.Generator(device=DEV).manual_seed(case)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    x, w = rn(T, in_dim).bfloat16(), (rn(out, in_dim) * in_dim ** -0.5).bfloat16()
    a = [(rn(S, r, in_dim) * in_dim ** -0.5).bfloat16() for _ in outs]
    b = [rn(S, o, r).bfloat16() for o in outs]
    cols = [sum(outs[:i]) for i in range(len(outs))]
    ranks = torch.tensor([r, 0, min(r, 8), r, r], dtype=torch.int32, device=DEV)
    for s in range(S):
        for t in a:
            t[s, int(ranks[s]):] = 0
        for t in b:
            t[s, :, int(ranks[s]):] = 0
    slots = torch.randint(-1, S, (T,), generator=torch.Generator().manual_seed(case), dtype=torch.int32)
    slots[T // 2:] = 3  # a popular adapter: several windows
    meta = metadata_for(slots, "graph", S)
    n = N.lib().lora_b200_decode_planes(in_dim, out)
    planes = torch.full((n, T, out), float("nan"), device=DEV)
    lora = (0, None, None, None, None, 0, 0, None, None, None, None, None, None, 0)
    if with_lora:
        lora = (len(outs), N.ptr_array(a), N.ptr_array(b), N.int_array(outs), N.int_array(cols), S, r, ranks.data_ptr(),
                meta.token_to_slot.data_ptr(), meta.token_indices_sorted_by_slot.data_ptr(), meta.active_slot_ids.data_ptr(),
                meta.num_tokens_per_slot.data_ptr(), meta.slot_start_offsets.data_ptr(), S + 1)
    N.check(N.lib().lora_b200_decode_linear(planes.data_ptr(), x.data_ptr(), in_dim, T, in_dim, w.data_ptr(), in_dim, out, *lora,
                                            N.current_stream(torch.device(DEV))))
    torch.cuda.synchronize()
    assert N.device_status(reset=True) == 0
    xd = x.double()
    # sums of in_dim products in fp32, in any order (the error of a sum is at most in_dim * 2^-24 of the sum of magnitudes, and grows like its root)
    base, base_mag = xd @ w.double().t(), xd.abs() @ w.double().abs().t()
    eps = 4 * in_dim ** 0.5 * 2 ** -24
    got = planes[: n - 1].double().sum(0)
    assert ((got - base).abs() <= eps * base_mag + 1e-30).all()
    if not with_lora:
        assert planes[n - 1].isnan().all(), "the plane of the delta is not the base product's to write"
        return
    delta, bound = torch.zeros_like(base), torch.zeros_like(base)
    for t in range(T):
        s = int(slots[t])
        if s < 0:
            continue
        for ai, bi, c, o in zip(a, b, cols, outs):
            tmp, bd = xd[t] @ ai[s].double().t(), bi[s].double()
            mag = xd[t].abs() @ ai[s].double().abs().t()
            delta[t, c:c + o] = bd @ tmp
            # the intermediate: fp32 sums, then one rounding to bf16 (8 significant bits: 2^-8 of the value at most), or to two such
            # numbers (2^-16) where r % 32 != 0
            bound[t, c:c + o] = bd.abs() @ ((2 ** -8 if r % 32 == 0 else 2 ** -16) * tmp.abs() + eps * mag) + 2 ** -20 * (bd.abs() @ tmp.abs())
    err = (planes[n - 1].double() - delta).abs()
    assert (err <= 1.01 * bound).all(), f"delta off by {(err / bound.clamp_min(1e-30)).max():.3g} of its bound"
    none = (slots < 0) | (slots == 1)
    assert not planes[n - 1][none.to(DEV)].any(), "rows without adapter must have a zero delta"


# heads, kv heads, head dim, planes, rotation table of the full or half width, its type, contexts (a warp takes blocks of 16 tokens, eight warps in turn)
ATTENTION = [
    (16, 2, 64, 9, False, torch.float32, [1, 2, 15, 16, 17, 129, 367, 368, 369, 800]),
    (4, 4, 64, 2, True, torch.bfloat16, [40, 736, 737]),
    (16, 1, 64, 1, False, torch.bfloat16, [5, 300]),
    (8, 2, 128, 5, True, torch.float32, [1, 16, 191, 192, 193, 384, 385, 500]),
    (32, 8, 128, 3, False, torch.float32, [64, 1000]),
    # a warp's blocks of 16 tokens: the first and last of a round of eight warps, of the three slots of a warp, one token more
    (16, 2, 64, 9, False, torch.float32, [111, 112, 113, 127, 128, 383, 384, 385, 400, 513]),
    (16, 2, 128, 9, False, torch.float32, [111, 113, 128, 130, 255, 256, 257, 400]),
]


@pytest.mark.parametrize("case", range(len(ATTENTION)))
def test_decode_attention(case):
    heads, kv, dim, n, full, table_dtype, ctx = ATTENTION[case]
    ctx = [0, *ctx]  # (a row that pads a graph's batch)
    T, block = len(ctx), 32
    gen = torch.Generator(device=DEV).manual_seed(case)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    planes = rn(n, T, (heads + 2 * kv) * dim) / n ** 0.5
    max_pos = 1024
    angle = torch.outer(torch.arange(max_pos, device=DEV).float(), 10000.0 ** (-torch.arange(0, dim, 2, device=DEV).float() / dim))
    angle = torch.cat((angle, angle), dim=1) if full else angle
    cos, sin = angle.cos().to(table_dtype), angle.sin().to(table_dtype)
    per = -(-max(ctx) // block)
    tables = torch.randperm(T * per + 3, generator=torch.Generator().manual_seed(case))[: T * per].to(torch.int32).view(T, per).to(DEV)
    k_cache, v_cache = (rn(T * per + 3, block, kv, dim).bfloat16() for _ in range(2))
    lens = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    pos = (lens.long() - 1).clamp_min(0)
    where = tables[torch.arange(T, device=DEV), pos // block].long() * block + pos % block
    where[0] = -1
    where[-1] = -1  # attended to, but stored nowhere
    before = k_cache.clone(), v_cache.clone()
    out = torch.full((T, heads * dim), 9.0, device=DEV, dtype=torch.bfloat16)
    N.check(N.lib().lora_b200_decode_attention(
        out.data_ptr(), planes.data_ptr(), n, T, heads, kv, dim, pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), cos.size(1),
        N.dtype_code(table_dtype), max_pos, k_cache.data_ptr(), v_cache.data_ptr(), tables.data_ptr(), per, block, lens.data_ptr(),
        where.data_ptr(), dim ** -0.5, N.current_stream(torch.device(DEV))))
    torch.cuda.synchronize()
    # q, k, v: planes added one after the other, products and sums of the rotation rounded one by one, then bf16: bit by bit
    row = torch.zeros_like(planes[0])
    for p in planes:
        row = row + p
    q, k, v = row.view(T, -1, dim).split([heads, kv, kv], dim=1)
    c, s = cos[pos].float().unsqueeze(1), sin[pos].float().unsqueeze(1)
    half = dim // 2
    turn = lambda t: torch.cat((t[..., :half] * c[..., :half] + -t[..., half:] * s[..., :half],  # noqa: E731
                                t[..., half:] * c[..., -half:] + t[..., :half] * s[..., -half:]), dim=-1)
    q, k, v = turn(q).bfloat16(), turn(k).bfloat16(), v.bfloat16()
    for new, old, mine in ((k_cache, before[0], k), (v_cache, before[1], v)):
        want = old.clone().view(-1, kv, dim)
        want[where[1:-1]] = mine[1:-1]
        assert torch.equal(new.view(-1, kv, dim), want), "cache rows"
    assert not out[0].any()
    for t in range(1, T):
        at = (tables[t].long()[:, None] * block + torch.arange(block, device=DEV)).view(-1)[: ctx[t]]
        kt, vt = before[0].view(-1, kv, dim)[at].clone(), before[1].view(-1, kv, dim)[at].clone()
        kt[-1], vt[-1] = k[t], v[t]
        kt, vt = (u.double().repeat_interleave(heads // kv, 1) for u in (kt, vt))
        p = (torch.einsum("hd,khd->hk", q[t].double(), kt) * dim ** -0.5).softmax(-1)
        ref, mag = torch.einsum("hk,khd->hd", p, vt).view(-1), torch.einsum("hk,khd->hd", p, vt.abs()).view(-1)
        # probabilities rounded to bf16 (2^-8 of each at most) ahead of the sum, the result once more; scores and sums in fp32
        bound = 2 ** -8 * (mag + ref.abs()) + 1e-4 * mag
        assert ((out[t].double() - ref).abs() <= 1.01 * bound).all(), f"context {ctx[t]}"
    assert N.device_status(reset=True) == 0


@pytest.mark.parametrize("shape", [(64, 1024, [1024, 128, 128], 16), (50, 512, [4096, 4096], 16), (90, 512, [1184, 96, 8], 48), (128, 2048, [2048], 80)],
                         ids=lambda s: f"{s[0]}x{s[1]}-r{s[3]}")
def test_planes_of_an_intermediate_of_two_numbers(shape, monkeypatch):
    """Ranks that are no multiple of 32 beside a GEMM: several output tiles a CTA, narrow ones among them."""
    monkeypatch.setitem(globals(), "LINEAR", [shape])
    test_decode_linear_planes(0, True)
