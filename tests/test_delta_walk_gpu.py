"""The gated delta rule as a walk over rows prepared in parallel (delta_tokens), against the token-by-token kernel on the same
projections: several segments of one pass, some behind a context, one idle, key and value sizes around what a lane, a warp and a
block hold. Both sum the same fp32 products in different orders: over D <= 256 terms and 70 tokens of a contracting recurrence their
results differ by a few times sqrt(D) 2^-24 of the largest, far below 1e-5; bf16 outputs by one rounding, 2^-8."""

import pytest
import torch

from nanochat_b200.mixers import ChannelDelta, RowPlan, Rows
from tests import rekudra_cases as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("sizes", [dict(dim=16, vdim=16, conv=1, heads=1, kv_heads=1), dict(dim=64, vdim=48, heads=4, kv_heads=2), dict(dim=80, vdim=272, heads=2, kv_heads=1),
                                   dict(dim=128, vdim=128, heads=3, kv_heads=3), dict(dim=144, vdim=32, conv=6, heads=2, kv_heads=2), dict(dim=256, vdim=64, conv=2, heads=2, kv_heads=1),
                                   # two and four values per lane at every number of key channels per lane, a last block of values that is not full
                                   dict(dim=64, vdim=128, heads=4, kv_heads=2), dict(dim=192, vdim=128, heads=4, kv_heads=4), dict(dim=256, vdim=128, heads=4, kv_heads=1),
                                   dict(dim=64, vdim=128, heads=8, kv_heads=4), dict(dim=128, vdim=144, heads=8, kv_heads=2), dict(dim=192, vdim=128, heads=8, kv_heads=8),
                                   dict(dim=256, vdim=128, heads=8, kv_heads=2)])
def test_walk_equals_token_by_token(dtype, sizes):
    entry, C = cases.delta(**sizes), 64
    state = cases.random_state(cases.config([entry], width=C), 61)
    mixer = ChannelDelta(entry["mixer"], {k[7:]: v for k, v in state.items() if k.startswith("l0.mix.")}, 1e-5, 128, dtype, "cuda")
    counts, starts, slots = [17, 1, 33, 4, 70], [0, 5, 2, 3, 0], [3, 0, 4, 1, 2]
    pos = [p if s != 1 else -1 for s, n, at in zip(slots, counts, starts) for p in range(at, at + n)]  # slot 1 is idle
    rows_slots = [s for s, n in zip(slots, counts) for _ in range(n)]
    plan_pos = [p for n, at in zip(counts, starts) for p in range(at, at + n)]
    n = len(pos)
    gen = torch.Generator(device="cuda").manual_seed(62)
    proj = torch.randn(n, mixer.in_width, generator=gen, device="cuda").to(dtype)
    found = []
    for walked_from in (2, 10 ** 9):
        mixer.WALKED_FROM, mixer.CHUNKED_FROM = walked_from, 10 ** 9
        cache, status = mixer.new_cache(5, 128), torch.zeros(1, dtype=torch.int32, device="cuda")
        gen.manual_seed(63)
        cache.state.state.normal_(generator=gen)
        cache.ring.rows.copy_(torch.randn(cache.ring.rows.shape, generator=gen, device="cuda"))
        out = torch.full((n, mixer.out_width), 7.0, dtype=dtype, device="cuda")
        mixer.run(proj, cache, Rows(n, torch.tensor(pos, dtype=torch.int32, device="cuda"), torch.tensor(rows_slots, dtype=torch.int32, device="cuda"), 128, status,
                                    RowPlan(rows_slots, plan_pos, "cuda")), out)
        assert int(status.item()) == 0
        found.append((out[:, :mixer.heads * mixer.vdim].double(), cache.state.state.double()))
    (out, last), (want, want_last) = found
    idle = torch.tensor([p < 0 for p in pos], device="cuda")
    assert not out[idle].any() and torch.equal(last[1], want_last[1])
    assert float((last - want_last).abs().max() / want_last.abs().max()) < 1e-5
    assert float((out - want).abs().max() / want.abs().max()) < (2 ** -8 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [1, 2, 3, 4, 6])
def test_a_sequence_that_is_not_finite_stays_alone(dtype, taps):
    """Sequences behind one that ends in infinities and NaN, from their start and behind a context: outputs and states bit for bit
    those of a pass without it, whatever the taps (a tap that does not exist has no row, not one of weight zero)."""
    entry, C = cases.delta(dim=32, vdim=32, heads=2, kv_heads=1, conv=taps), 64
    state = cases.random_state(cases.config([entry], width=C), 64)
    mixer = ChannelDelta(entry["mixer"], {k[7:]: v for k, v in state.items() if k.startswith("l0.mix.")}, 1e-5, 128, dtype, "cuda")
    mixer.WALKED_FROM, mixer.CHUNKED_FROM = 2, 10 ** 9
    runs = [(0, 0, 19), (1, 0, 9), (2, 5, 14)]  # slot, first position, rows
    slots, pos = [s for s, _, n in runs for _ in range(n)], [p for _, at, n in runs for p in range(at, at + n)]
    gen = torch.Generator(device="cuda").manual_seed(65)
    proj = torch.randn(len(pos), mixer.in_width, generator=gen, device="cuda").to(dtype)
    proj[16:19], proj[17] = float("inf"), float("nan")
    found = []
    for first in (0, 19):
        cache, status = mixer.new_cache(3, 64), torch.zeros(1, dtype=torch.int32, device="cuda")
        gen.manual_seed(66)
        cache.state.state.normal_(generator=gen)
        cache.ring.rows.copy_(torch.randn(cache.ring.rows.shape, generator=gen, device="cuda"))
        part, n = proj[first:].contiguous(), len(pos) - first
        out = torch.zeros((n, mixer.out_width), dtype=dtype, device="cuda")
        mixer.run(part, cache, Rows(n, torch.tensor(pos[first:], dtype=torch.int32, device="cuda"), torch.tensor(slots[first:], dtype=torch.int32, device="cuda"), 64,
                                    status, RowPlan(slots[first:], pos[first:], "cuda")), out)
        assert int(status.item()) == 0
        found.append((out[19 - first:], cache.state.state[1:]))
    (out, last), (want, want_last) = found
    assert bool(torch.isfinite(want.float()).all()) and torch.equal(out, want) and torch.equal(last, want_last)
