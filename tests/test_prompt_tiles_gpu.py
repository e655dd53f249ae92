"""Prompt attention on tcgen05 (csrc/attn_tiles.cuh) against float64 on the same operands and beside the kernels on mma.sync: runs of
rows around the edges of a row tile (128) and a key tile (64), behind contexts of none, one and many keys, with NaN wherever the
cache holds nothing. An output is one bf16 rounding (2^-9) of a sum whose weights carry 16 bits (11 over the fp8 cache)."""

import ctypes

import pytest
import torch

import nanochat_b200 as ncb
from nanochat_b200 import attention as ops
from nanochat_b200.mixers import ChannelDelta, GroupedAttention, LatentAttention, RowPlan, Rows
from nanochat_b200.native import Conv, Gqa, Latent, check, cuda_library, stream
from tests import pudisun_cases, rekudra_cases

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64
NCB_DEV_BAD_LENGTH = 4
RUNS = [[(0, 1)], [(0, 64), (7, 63)], [(0, 65), (63, 130)], [(1, 127), (0, 128), (64, 129)], [(300, 257)], [(0, 700), (1000, 3), (5, 90)]]


def attended(q, k, v, scale, start, sink=None):
    """float64: q [n, H, D] at positions start .., k, v [H, start + n, ..] -> [n, H, V]; sink: logits of a key without a value."""
    n, N = q.shape[0], k.shape[1]
    s = torch.einsum("nhd,hkd->hnk", q.to(F64), k.to(F64)) * scale
    seen = torch.arange(N, device=q.device)[None, :] <= torch.arange(start, start + n, device=q.device)[:, None]
    s = s.masked_fill(~seen, float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink.to(F64)[:, None, None].expand(-1, n, 1)], 2)
    return torch.einsum("hnk,hkv->nhv", s.softmax(-1)[..., :N], v.to(F64))


def off(got, want):
    return float((got.to(F64) - want).norm() / want.norm())


def judged(found, want):
    """The new kernel within bf16's rounding of the value, and no further from it than the old one (rounding noise aside)."""
    new, old = found
    assert torch.isfinite(new.float()).all()
    assert off(new, want) < 2 ** -8 and off(new, want) <= 1.05 * off(old, want) + 1e-6, (off(new, want), off(old, want))
    assert float((new.to(F64) - want).abs().max()) <= 2 ** -7 * float(want.abs().max())


@pytest.mark.parametrize("runs", RUNS, ids=str)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 4, 128, 128), (6, 2, 128, 64), (4, 1, 64, 128), (2, 2, 64, 64)])
def test_grouped(heads, kv_heads, dim, vdim, runs):
    gen = torch.Generator(device="cuda").manual_seed(70)
    slots, pos = [s for s, (_, n) in enumerate(runs) for _ in range(n)], [p for at, n in runs for p in range(at, at + n)]
    n, capacity, scale = len(pos), 1088, 2.0 * dim ** -0.5
    q = torch.randn(n, heads, dim, generator=gen, device="cuda").to(BF16)
    kv = torch.full((len(runs), kv_heads, capacity, dim + vdim), float("nan"), dtype=BF16, device="cuda")
    for s, (at, count) in enumerate(runs):
        kv[s, :, :at + count] = torch.randn(kv_heads, at + count, dim + vdim, generator=gen, device="cuda").to(BF16)
        kv[s, :, :at + count, :dim] *= (1 + (torch.arange(at + count, device="cuda") % 97 == 96))[None, :, None]  # maxima that move late
    ldp = heads * dim  # the projection's rows: only the gate is read
    proj = torch.randn(n, ldp, generator=gen, device="cuda").to(BF16)
    dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slots)]
    status, plan, lib, found = torch.zeros(1, dtype=torch.int32, device="cuda"), RowPlan(slots, pos, "cuda"), cuda_library("gqa_attn"), []
    ring, taps = torch.zeros(len(runs), 1, ldp, dtype=BF16, device="cuda"), torch.ones(1, ldp, device="cuda")
    for wide in (True, False):
        out = torch.full((n, heads * vdim + 8), 7.0, dtype=BF16, device="cuda")
        a = Gqa(conv=Conv(proj=proj.data_ptr(), ring=ring.data_ptr(), w=taps.data_ptr(), rows=n, ldp=ldp, taps=1, width=ldp, n_slots=len(runs),
                          pos=dev[0].data_ptr(), slot_map=dev[1].data_ptr()), q=q.data_ptr(), kv=kv.data_ptr(), out=out.data_ptr(), ldo=out.stride(0),
                heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, norm_count=dim, capacity=capacity, table_len=capacity, scale=scale, eps=1e-6,
                status=status.data_ptr())
        tiles, a.n_tiles = plan.row_tiles(128 if wide else 64)
        a.tile_row, a.tile_rows, a.tile_pos = (tiles[i].data_ptr() for i in (0, 1, 3))
        check((lib.gqa_prefill_tiles if wide else lib.gqa_prefill)(ctypes.byref(a), stream()), "gqa")
        assert int(status.item()) == 0 and bool((out[:, heads * vdim:] == 7.0).all())
        found.append(out[:, :heads * vdim].view(n, heads, vdim))
    want, row = [], 0
    for s, (at, count) in enumerate(runs):
        k, v = (t.repeat_interleave(heads // kv_heads, 0) for t in kv[s, :, :at + count].split([dim, vdim], -1))
        want.append(attended(q[row:row + count], k, v, scale, at) * torch.sigmoid(proj[row:row + count, :heads].to(F64))[..., None])
        row += count
    judged(found, torch.cat(want))


@pytest.mark.parametrize("runs", RUNS, ids=str)
@pytest.mark.parametrize("heads,dim,vdim,sink,gated", [(3, 128, 128, True, True), (2, 128, 64, False, False), (2, 64, 128, True, False), (2, 64, 64, False, True)])
def test_latent(heads, dim, vdim, sink, gated, runs):
    gen, rot = torch.Generator(device="cuda").manual_seed(71), 64
    slots, pos = [s for s, (_, n) in enumerate(runs) for _ in range(n)], [p for at, n in runs for p in range(at, at + n)]
    n, contexts = len(pos), [at + count for at, count in runs]
    ldp, ld, scale = heads * (dim + rot + vdim) + 8, heads * (dim + vdim) + 64, 2.0 * (dim + rot) ** -0.5
    proj = torch.randn(n, ldp, generator=gen, device="cuda").to(BF16)
    kv, kr = (torch.randn(sum(contexts), w, generator=gen, device="cuda").to(BF16) for w in (ld, rot))
    sinks = torch.randn(heads, generator=gen, device="cuda")
    dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slots)]
    some = torch.ones(64, device="cuda")
    status, plan, lib, found = torch.zeros(1, dtype=torch.int32, device="cuda"), RowPlan(slots, pos, "cuda"), cuda_library("latent_attn"), []
    for wide in (True, False):
        out = torch.full((n, heads * vdim + 8), 7.0, dtype=BF16, device="cuda")
        a = Latent(proj=proj.data_ptr(), cache=kv.data_ptr(), out=out.data_ptr(), rows=n, ldp=ldp, ldo=out.stride(0), off_g=heads * (dim + rot), gated=int(gated),
                   heads=heads, dim=dim, rot=rot, vdim=vdim, rank=32, norm_count=32, n_slots=len(runs), capacity=2000, table_len=2000, scale=scale,
                   eps=1e-6, norm=some.data_ptr(), cos=some.data_ptr(), sin=some.data_ptr(), sink=sinks.data_ptr() if sink else None,
                   pos=dev[0].data_ptr(), slot_map=dev[1].data_ptr(), ctx_rot=kr.data_ptr(), ctx_kv=kv.data_ptr(), ctx_kv_ld=ld, status=status.data_ptr())
        tiles, a.n_tiles = plan.row_tiles(128 if wide else 64)
        a.tile_row, a.tile_rows, a.tile_ctx, a.tile_pos = (t.data_ptr() for t in tiles)
        check(lib.latent_prefill_tiles(ctypes.byref(a), sum(contexts), stream()) if wide else lib.latent_prefill(ctypes.byref(a), stream()), "latent")
        assert int(status.item()) == 0 and bool((out[:, heads * vdim:] == 7.0).all())
        found.append(out[:, :heads * vdim].view(n, heads, vdim))
    want, row, first = [], 0, 0
    for (at, count), length in zip(runs, contexts):
        both = kv[first:first + length, :heads * (dim + vdim)].view(length, heads, dim + vdim).transpose(0, 1)
        k = torch.cat([both[..., :dim], kr[first:first + length].expand(heads, -1, -1)], -1)
        part = proj[row:row + count]
        o = attended(part[:, :heads * (dim + rot)].view(count, heads, dim + rot), k, both[..., dim:], scale, at, sinks if sink else None)
        if gated:
            o = o * torch.sigmoid(part[:, heads * (dim + rot):heads * (dim + rot + vdim)].to(F64)).view(count, heads, vdim)
        want.append(o)
        row, first = row + count, first + length
    judged(found, torch.cat(want))


@pytest.mark.parametrize("runs", RUNS, ids=str)
@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (8, 2), (16, 1), (6, 2)])
def test_fp8(Hq, Hkv, runs):
    gen = torch.Generator(device="cuda").manual_seed(72)
    lens = [at + n for at, n in runs]
    cache = ncb.Fp8KVCache(len(runs), Hkv, max(lens) + 70)
    kept = []
    for s, n in enumerate(lens):
        rows = [torch.randn(Hkv, cache.capacity, 128, generator=gen, device="cuda") * torch.rand(Hkv, cache.capacity, 1, generator=gen, device="cuda").mul_(4).exp2() for _ in "kv"]
        rows[1][:, 1 + n // 2] = 0.0  # a value of zeros: its scale is zero
        made = []
        for t in rows:
            scale = t.abs().amax(-1) / 448.0
            b = (t / scale.clamp(min=1e-30)[..., None]).to(torch.float8_e4m3fn)
            made.append((b.view(torch.uint8).clone(), scale, b.to(F64) * scale[..., None].to(F64)))
            made[-1][0][:, n:], scale[:, n:] = 0x7f, float("nan")
        cache.write(s, made[0][0], made[0][1], made[1][0], made[1][1])
        kept.append([m[2][:, :n].repeat_interleave(Hq // Hkv, 0) for m in made])
    slots, pos = [s for s, (_, n) in enumerate(runs) for _ in range(n)], [p for at, n in runs for p in range(at, at + n)]
    q = torch.randn(len(pos), Hq, 128, generator=gen, device="cuda").to(BF16)
    status, found = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    plan = ops.PrefillPlan(slots, pos, Hq, cache, "cuda", widen=True)  # the choice is not what is tested here
    assert plan.wide is not None
    for wide in (plan.wide, None):
        plan.wide = wide
        found.append(ops.prefill_attention(q, cache, plan, status=status))
        assert int(status.item()) == 0
    want, row = [], 0
    for (at, n), (k, v) in zip(runs, kept):
        want.append(attended(q[row:row + n], k, v, 128 ** -0.5, at))
        row += n
    judged(found, torch.cat(want))


def test_fp8_rows_without_a_finite_score_are_zero():
    """A query that is NaN, and a first position whose key is: nothing to attend, zeros, in both kernels."""
    gen, n = torch.Generator(device="cuda").manual_seed(77), 200
    cache = ncb.Fp8KVCache(1, 2, 256)
    raw, scale = torch.randn(2, 256, 128, generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8), torch.ones(2, 256, device="cuda")
    first = scale.clone()
    first[1, 0] = float("nan")
    cache.write(0, raw, first, raw, scale)
    q = torch.randn(n, 4, 128, generator=gen, device="cuda").to(BF16)
    q[70, 1] = float("nan")
    status, found = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    plan = ops.PrefillPlan([0] * n, list(range(n)), 4, cache, "cuda", widen=True)
    for wide in (plan.wide, None):
        plan.wide = wide
        found.append(ops.prefill_attention(q, cache, plan, status=status))
        assert int(status.item()) == 0
        assert not found[-1][70, 1].any() and not found[-1][0, 2:].any()
        assert bool(torch.isfinite(found[-1][:, :2].float()).all()) and bool(torch.isnan(found[-1][1:, 2:].float()).all())
    assert off(found[0][:, :2], found[1][:, :2].double()) < 2 ** -7


def test_fp8_route():
    """Where the widened form does not apply the plan has none: short runs, a workspace beyond its bound, rows outside the cache."""
    cache = ncb.Fp8KVCache(2, 2, 1024)
    plan = lambda slots, pos, Hq=4: ops.PrefillPlan(slots, pos, Hq, cache, "cuda").wide  # noqa: E731
    assert plan([0] * 700, list(range(700))) is not None and plan([0] * 300, list(range(300))) is not None
    assert plan([0] * 150, list(range(150))) is None and plan([0] * 63, list(range(900, 963))) is None
    assert plan([0] * 700, list(range(400, 1100))) is None and plan([2] * 700, list(range(700))) is None
    assert plan([0] * 700, list(range(-1, 699))) is None
    bound = ops.PrefillPlan.WIDE_BYTES
    try:
        ops.PrefillPlan.WIDE_BYTES = 1000
        assert plan([0] * 700, list(range(700))) is None
    finally:
        ops.PrefillPlan.WIDE_BYTES = bound


def test_fp8_pages_outside_the_cache_are_flagged_and_not_read():
    """A plan used with a cache of fewer slots, or of fewer pages: what lies outside is flagged and its rows are zero, as in a pass
    that never had widened pages; the library on its own flags the pages, does not read them and takes zeros in their place."""
    gen = torch.Generator(device="cuda").manual_seed(74)
    large = ncb.Fp8KVCache(3, 2, 512)
    raw = torch.randn(3, 2, 512, 128, generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    ones = torch.ones(2, 512, device="cuda")
    for s in range(3):
        large.write(s, raw[s], ones, raw[s], ones)
    for n_slots, capacity in ((1, 512), (2, 512), (3, 256), (2, 384)):
        small = ncb.Fp8KVCache(n_slots, 2, capacity)
        small.pages.copy_(large.pages[:n_slots, :, :small.pages_per_slot])
        runs = [(0, 200), (1, 384), (2, 300)]
        slots, pos = [s for s, n in runs for _ in range(n)], [p for _, n in runs for p in range(n)]
        plan = ops.PrefillPlan(slots, pos, 4, large, "cuda", widen=True)
        q = torch.randn(len(pos), 4, 128, generator=gen, device="cuda").to(BF16)
        status, fine = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
        out, tiles = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
        want = ops.prefill_attention(q, large, plan, status=fine)
        ops.prefill_attention(q, small, plan, out=out, status=status)
        assert int(fine.item()) == 0 and int(status.item()) == NCB_DEV_BAD_LENGTH
        status.zero_()
        plan.needs = (0, 0)  # past the check: the library's own
        ops.prefill_attention(q, small, plan, out=tiles, status=status)
        assert int(status.item()) == NCB_DEV_BAD_LENGTH and bool(torch.isfinite(tiles.float()).all())
        row = 0
        for s, n in runs:
            if s < n_slots and n <= capacity:
                assert off(out[row:row + n], want[row:row + n].double()) < 2 ** -7 and torch.equal(tiles[row:row + n], want[row:row + n])
            elif s >= n_slots:
                assert not out[row:row + n].any() and not tiles[row:row + n].any()
            else:
                assert not out[row + n - 22:row + n].any()  # at least the last block of rows
            row += n


# (first position, rows) and where a value, key or scale is not finite: early, late and at the borders of a tile of the run
PLANTED = [((0, 40), 5), ((0, 128), 127), ((0, 130), 64), ((63, 128), 100), ((62, 128), 130), ((200, 300), 430), ((200, 300), 201), ((7, 90), 96), ((0, 200), 0)]


def split_at(got, clean, row, columns):
    """Rows before `row` and all other columns as without the planted value, the rest not finite."""
    rest = [c for c in range(clean.shape[-1]) if c not in columns]
    assert torch.isfinite(got[:row].float()).all() and torch.isfinite(got[..., rest].float()).all()
    assert row == 0 or off(got[:row], clean[:row]) < 2 ** -8
    assert not rest or off(got[..., rest], clean[..., rest]) < 2 ** -8
    assert not torch.isfinite(got[row:][..., columns].float()).any()


@pytest.mark.parametrize("run,at", PLANTED, ids=str)
@pytest.mark.parametrize("vdim,bad", [(64, float("nan")), (128, float("inf"))])
def test_a_value_that_is_not_finite_reaches_only_rows_that_see_it(run, at, vdim, bad):
    """Grouped and latent attention: one value of one position is infinite or NaN."""
    gen, (start, n), heads, dim, rot = torch.Generator(device="cuda").manual_seed(75), run, 2, 128, 64
    length, plan, status = start + n, RowPlan([0] * n, list(range(start, start + n)), "cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    pos, slots = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (range(start, start + n), [0] * n))
    tiles, n_tiles = plan.row_tiles(128)
    row, column = max(at - start, 0), 3
    # grouped
    q, kv = torch.randn(n, heads, dim, generator=gen, device="cuda").to(BF16), torch.randn(heads, 512, dim + vdim, generator=gen, device="cuda").to(BF16)
    kv[:, length:] = float("nan")
    clean = kv[:, :length].clone()
    kv[:, at, dim + column] = bad
    proj, ring, taps = torch.zeros(n, heads * dim, dtype=BF16, device="cuda"), torch.zeros(1, 1, heads * dim, dtype=BF16, device="cuda"), torch.ones(1, heads * dim, device="cuda")
    out = torch.zeros((n, heads * vdim), dtype=BF16, device="cuda")
    a = Gqa(conv=Conv(proj=proj.data_ptr(), ring=ring.data_ptr(), w=taps.data_ptr(), rows=n, ldp=heads * dim, taps=1, width=heads * dim, n_slots=1,
                      pos=pos.data_ptr(), slot_map=slots.data_ptr()), q=q.data_ptr(), kv=kv.data_ptr(), out=out.data_ptr(), ldo=heads * vdim, heads=heads, kv_heads=heads,
            dim=dim, vdim=vdim, norm_count=dim, capacity=512, table_len=512, scale=0.1, eps=1e-6, status=status.data_ptr(), n_tiles=n_tiles)
    a.tile_row, a.tile_rows, a.tile_pos = (tiles[i].data_ptr() for i in (0, 1, 3))
    check(cuda_library("gqa_attn").gqa_prefill_tiles(ctypes.byref(a), stream()), "gqa_prefill_tiles")
    assert int(status.item()) == 0
    split_at(out.view(n, heads, vdim), 0.5 * attended(q, clean[..., :dim], clean[..., dim:], 0.1, start), row, [column])
    # latent
    width, ld = dim + rot, heads * (dim + vdim)
    proj, ctx, kr = (torch.randn(m, w, generator=gen, device="cuda").to(BF16) for m, w in ((n, heads * width), (length, ld), (length, rot)))
    both = ctx.view(length, heads, dim + vdim).transpose(0, 1).clone()
    ctx.view(length, heads, dim + vdim)[at, :, dim + column] = bad
    out, some = torch.zeros((n, heads * vdim), dtype=BF16, device="cuda"), torch.ones(64, device="cuda")
    a = Latent(proj=proj.data_ptr(), cache=ctx.data_ptr(), out=out.data_ptr(), rows=n, ldp=heads * width, ldo=heads * vdim, heads=heads, dim=dim, rot=rot, vdim=vdim,
               rank=32, norm_count=32, n_slots=1, capacity=512, table_len=512, scale=0.1, eps=1e-6, norm=some.data_ptr(), cos=some.data_ptr(), sin=some.data_ptr(),
               pos=pos.data_ptr(), slot_map=slots.data_ptr(), ctx_rot=kr.data_ptr(), ctx_kv=ctx.data_ptr(), ctx_kv_ld=ld, status=status.data_ptr(), n_tiles=n_tiles)
    a.tile_row, a.tile_rows, a.tile_ctx, a.tile_pos = (t.data_ptr() for t in tiles)
    check(cuda_library("latent_attn").latent_prefill_tiles(ctypes.byref(a), length, stream()), "latent_prefill_tiles")
    assert int(status.item()) == 0
    want = attended(proj.view(n, heads, width), torch.cat([both[..., :dim], kr.expand(heads, -1, -1)], -1), both[..., dim:], 0.1, start)
    split_at(out.view(n, heads, vdim), want, row, [column])


@pytest.mark.parametrize("run,at", PLANTED, ids=str)
@pytest.mark.parametrize("what", ["value", "value's scale", "key's scale"])
def test_fp8_position_that_is_not_finite_reaches_only_rows_that_see_it(run, at, what):
    gen, (start, n), Hkv = torch.Generator(device="cuda").manual_seed(76), run, 2
    length = start + n
    cache = ncb.Fp8KVCache(1, Hkv, 512)
    raw = torch.randn(2, Hkv, 512, 128, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    scale = torch.rand(2, Hkv, 512, generator=gen, device="cuda") + 0.5
    k, v = (raw[i, :, :length].to(F64) * scale[i, :, :length, None].to(F64) for i in (0, 1))
    b, columns, row = raw.view(torch.uint8).clone(), list(range(128)), max(at - start, 0)
    b[:, :, length:], scale[:, :, length:] = 0x7f, float("nan")
    if what == "value":
        b[1, :, at, 3], columns = 0x7f, [3]
    else:
        scale[int(what[0] == "v"), :, at] = float("nan") if at % 2 else float("inf")
    cache.write(0, b[0], scale[0], b[1], scale[1])
    q = torch.randn(n, 4, 128, generator=gen, device="cuda").to(BF16)
    status, plan = torch.zeros(1, dtype=torch.int32, device="cuda"), ops.PrefillPlan([0] * n, list(range(start, length)), 4, cache, "cuda", widen=True)
    assert plan.wide is not None
    got = ops.prefill_attention(q, cache, plan, softmax_scale=0.1, status=status)
    assert int(status.item()) == 0
    want = attended(q, k.repeat_interleave(2, 0), v.repeat_interleave(2, 0), 0.1, start)
    rows = row if what == "key's scale" else n  # (rows that see such a key: NaN, or its value where it is the only one of weight)
    split_at(got[:rows], want[:rows], row, columns)


def mixer_of(kind: str):
    """A mixer whose prompts run on tcgen05 (or as a walk), with random weights."""
    if kind == "latent":
        entry = pudisun_cases.latent(heads=2, dim=128, rot_dim=64, vdim=128)
        state = pudisun_cases.random_state(pudisun_cases.config([entry], width=64), 81)
    else:
        entry = rekudra_cases.attention(heads=4, kv_heads=2, dim=128, vdim=128, rot_dims=32) if kind == "grouped" else rekudra_cases.delta(dim=64, vdim=64)
        state = rekudra_cases.random_state(rekudra_cases.config([entry], width=64), 81)
    cls = {"latent": LatentAttention, "grouped": GroupedAttention, "delta": ChannelDelta}[kind]
    mixer = cls(entry["mixer"], {k[7:]: v for k, v in state.items() if k.startswith("l0.mix.")}, 1e-5, 128, BF16, "cuda")
    mixer.expands = lambda plan: True
    return mixer


def run_counts(mixer, counts, proj, out=None):
    """Segments of `counts` rows, each a slot of its own from position 0, through the mixer."""
    slots, pos = [s for s, n in enumerate(counts) for _ in range(n)], [p for n in counts for p in range(n)]
    status, n = torch.zeros(1, dtype=torch.int32, device="cuda"), len(pos)
    out = torch.zeros((n, mixer.out_width), dtype=BF16, device="cuda") if out is None else out
    dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slots)]
    mixer.run(proj.clone(), mixer.new_cache(len(counts), 512), Rows(n, *dev, max(counts), status, RowPlan(slots, pos, "cuda")), out)
    assert int(status.item()) == 0
    return out


@pytest.mark.parametrize("kind,off_by", [("latent", 2), ("grouped", 2), ("delta", 1), ("delta", 8)])
def test_outputs_that_are_not_in_chunks_of_16_bytes(kind, off_by):
    """Rows at a stride (or projections at one) that the kernels on tcgen05 and the walk do not take: the other kernels', bit for bit."""
    mixer, counts = mixer_of(kind), [40, 17]
    proj = torch.randn(sum(counts), mixer.in_width, generator=torch.Generator(device="cuda").manual_seed(82), device="cuda").to(BF16)
    mixer.CHUNKED_FROM = 10 ** 9
    out = torch.zeros((sum(counts), mixer.out_width + off_by), dtype=BF16, device="cuda")[:, :mixer.out_width]
    found = run_counts(mixer, counts, proj, out)
    if off_by % 8:
        mixer.wide = mixer.walks = False
    assert torch.equal(found, run_counts(mixer, counts, proj))


@pytest.mark.parametrize("kind", ["latent", "grouped"])
def test_a_segments_length_chooses_its_kernel(kind):
    """Long and short segments in one pass: every one as in a pass of its own, bit for bit."""
    mixer, counts = mixer_of(kind), [200, 10, 40, 15, 31, 16, 32, 130, 8]
    proj = torch.randn(sum(counts), mixer.in_width, generator=torch.Generator(device="cuda").manual_seed(83), device="cuda").to(BF16)
    together, row = run_counts(mixer, counts, proj), 0
    for n in counts:
        assert torch.equal(together[row:row + n], run_counts(mixer, [n], proj[row:row + n])), n
        row += n


@pytest.mark.parametrize("runs", [[(0, 1)], [(0, 8), (3, 9)], [(31, 7), (32, 16), (25, 8)], [(300, 45), (0, 130)]], ids=str)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 4, 128, 128), (6, 2, 16, 48), (2, 1, 80, 256)])
def test_grouped_in_32_bits(heads, kv_heads, dim, vdim, runs):
    """gqa_prefill_f32 around the edges of its tiles of 8 rows and 32 keys, with NaN behind each sequence's end and infinities in the values
    of its last position, against float64: a sum of at most 345 weighted values and 128 products per score, a few times sqrt(345) 2^-24
    of the result's size; infinities only where the last position is seen."""
    gen = torch.Generator(device="cuda").manual_seed(75)
    slots, pos = [s for s, (_, n) in enumerate(runs) for _ in range(n)], [p for at, n in runs for p in range(at, at + n)]
    n, capacity, scale = len(pos), 384, dim ** -0.5
    ldp = heads * dim  # the projection's rows: only the gate is read
    q, proj = torch.randn(n, heads, dim, generator=gen, device="cuda"), torch.randn(n, ldp, generator=gen, device="cuda")
    gate = proj[:, :heads]
    kv = torch.full((len(runs), kv_heads, capacity, dim + vdim), float("nan"), device="cuda")
    for s, (at, count) in enumerate(runs):
        kv[s, :, :at + count] = torch.randn(kv_heads, at + count, dim + vdim, generator=gen, device="cuda")
        if at + count > 1:
            kv[s, :, at + count - 1, dim:] = float("inf")
    dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slots)]
    status, plan, lib = torch.zeros(1, dtype=torch.int32, device="cuda"), RowPlan(slots, pos, "cuda"), cuda_library("gqa_attn")
    ring, taps = torch.zeros(len(runs), 1, ldp, device="cuda"), torch.ones(1, ldp, device="cuda")
    out = torch.full((n, heads * vdim + 8), 7.0, device="cuda")
    a = Gqa(conv=Conv(proj=proj.data_ptr(), ring=ring.data_ptr(), w=taps.data_ptr(), rows=n, ldp=ldp, taps=1, width=ldp, n_slots=len(runs),
                      pos=dev[0].data_ptr(), slot_map=dev[1].data_ptr()), q=q.data_ptr(), kv=kv.data_ptr(), out=out.data_ptr(), ldo=out.stride(0),
            heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, norm_count=dim, capacity=capacity, table_len=capacity, scale=scale, eps=1e-6,
            status=status.data_ptr())
    tiles, a.n_tiles = plan.row_tiles(8)
    a.tile_row, a.tile_rows, a.tile_pos = (tiles[i].data_ptr() for i in (0, 1, 3))
    check(lib.gqa_prefill_f32(ctypes.byref(a), stream()), "gqa_prefill_f32")
    assert int(status.item()) == 0 and bool((out[:, heads * vdim:] == 7.0).all())
    got, row = out[:, :heads * vdim].view(n, heads, vdim), 0
    for s, (at, count) in enumerate(runs):
        k, v = (t.repeat_interleave(heads // kv_heads, 0) for t in kv[s, :, :at + count].split([dim, vdim], -1))
        seen = count - 1 if at + count > 1 else count  # rows that do not see the infinite values
        if seen:
            want = attended(q[row:row + seen], k[:, :at + seen], v[:, :at + seen], scale, at) * torch.sigmoid(gate[row:row + seen].to(F64))[..., None]
            assert float((got[row:row + seen].to(F64) - want).abs().max() / want.abs().max()) < 5e-6
        if seen < count:
            assert not torch.isfinite(got[row + count - 1]).any()
        row += count


def test_grouped_in_32_bits_answers_the_rows_before_a_refused_one():
    """A portion that runs over the end of the rotary table: rows up to it are what they are without the others, the rest are zeros and flagged."""
    gen = torch.Generator(device="cuda").manual_seed(76)
    heads, kv_heads, dim, vdim, capacity, table = 4, 2, 32, 48, 192, 133
    ldp, pos = heads * dim, list(range(120, 141))
    n, good = len(pos), table - 120
    q, proj = torch.randn(n, heads, dim, generator=gen, device="cuda"), torch.randn(n, ldp, generator=gen, device="cuda")
    kv = torch.randn(2, kv_heads, capacity, dim + vdim, generator=gen, device="cuda")
    ring, taps, lib = torch.zeros(2, 1, ldp, device="cuda"), torch.ones(1, ldp, device="cuda"), cuda_library("gqa_attn")

    def attend(count, slot):
        dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos[:count], [slot] * count)]
        status, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((count, heads * vdim), 7.0, device="cuda")
        a = Gqa(conv=Conv(proj=proj.data_ptr(), ring=ring.data_ptr(), w=taps.data_ptr(), rows=count, ldp=ldp, taps=1, width=ldp, n_slots=2,
                          pos=dev[0].data_ptr(), slot_map=dev[1].data_ptr()), q=q.data_ptr(), kv=kv.data_ptr(), out=out.data_ptr(), ldo=out.stride(0),
                heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, norm_count=dim, capacity=capacity, table_len=table, scale=dim ** -0.5, eps=1e-6,
                status=status.data_ptr())
        tiles, a.n_tiles = RowPlan([slot] * count, pos[:count], "cuda").row_tiles(8)
        a.tile_row, a.tile_rows, a.tile_pos = (tiles[i].data_ptr() for i in (0, 1, 3))
        check(lib.gqa_prefill_f32(ctypes.byref(a), stream()), "gqa_prefill_f32")
        return out, int(status.item())

    want, flags = attend(good, 1)
    assert flags == 0 and bool(want.any())
    got, flags = attend(n, 1)
    assert flags != 0 and torch.equal(got[:good], want) and not got[good:].any()
    got, flags = attend(n, 2)  # a slot that is not there
    assert flags != 0 and not got.any()
