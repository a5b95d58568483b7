"""The host's plan for the tcgen05 attention kernel (no GPU): tiles, their parts, and the schedule that deals the work
units out to the kernel's CTAs.  The library is loaded for its host-side functions only."""
import random

import pytest
import torch

from qwen_engine_b200 import ops

GEOS = [(16, 8, 128, 0), (4, 2, 128, 0), (8, 1, 128, 0), (4, 4, 128, 300)]


def _items(plan, key="tc0_items"):
    flat = plan[key]
    return [flat[i:i + ops.FLASH_ITEM_INTS] for i in range(0, len(flat), ops.FLASH_ITEM_INTS)]


def _random_batch(rng):
    n = rng.randint(1, 6)
    q_lens = [rng.choice([70, 128, 129, 300, 700, 1500, 2048, 3000]) for _ in range(n)]
    ctx_lens = [rng.choice([0, 0, 17, 128, 1000, 5000]) for _ in range(n)]
    return q_lens, ctx_lens


@pytest.mark.parametrize("seed", range(12))
def test_tiles_and_parts_cover_every_row_and_key_once(seed):
    rng = random.Random(seed)
    Hq, Hkv, D, window = GEOS[seed % len(GEOS)]
    q_lens, ctx_lens = _random_batch(rng)
    plan = ops.plan_attention(q_lens, ctx_lens, 16, ((Hq, Hkv, D, window),), torch.bfloat16)
    G = Hq // Hkv
    tile_tokens = ops.TC_ROWS // G
    seen = {}                                           # (request, first token of the tile) -> key ranges of its items
    for req, q0, lo, hi, part, n_parts, split, row0, q_len, ctx, _, _ in _items(plan):
        assert q_len == q_lens[req] and ctx == ctx_lens[req] and q0 % tile_tokens == 0 and q0 < q_len
        assert row0 == sum(q_lens[:req])
        seen.setdefault((req, q0), []).append((lo, hi, part, n_parts, split))
    for req, n in enumerate(q_lens):
        if n * G < ops.TC_MIN_ROWS:
            assert not any(r == req for r, _ in seen), "a request of few rows belongs to the other kernel"
            continue
        assert sorted(q0 for r, q0 in seen if r == req) == list(range(0, n, tile_tokens))
    for (req, q0), ranges in seen.items():
        ranges.sort()
        frontier = ctx_lens[req] + min(q_lens[req], q0 + tile_tokens)
        assert ranges[-1][1] == frontier, "a tile's keys end at its last token's position"
        if len(ranges) == 1:
            assert ranges[0][2] == -1 and ranges[0][0] >= 0
            continue
        first = ranges[0][2]
        for i, (lo, hi, part, n_parts, split) in enumerate(ranges):
            assert (part, n_parts, split) == (first + i, len(ranges), i)
            assert lo < hi and (i == 0 or lo == ranges[i - 1][1]), "the parts of a tile follow one another"
            assert i == 0 or lo % ops.TC_BN == 0, "a part begins with a whole key step"
    assert plan["tc0_info"][0] == sum(len(r) for r in seen.values() if len(r) > 1)


@pytest.mark.parametrize("seed", range(12))
@pytest.mark.parametrize("ctas", [1, 5, 148])
def test_every_unit_is_dealt_out_once_and_no_cta_is_left_behind(seed, ctas, monkeypatch):
    rng = random.Random(100 + seed)
    Hq, Hkv, D, window = GEOS[seed % len(GEOS)]
    q_lens, ctx_lens = _random_batch(rng)
    monkeypatch.setattr(ops, "TC_TARGET_CTAS", ctas)
    plan = ops.plan_attention(q_lens, ctx_lens, 16, ((Hq, Hkv, D, window),), torch.bfloat16)
    if "tc0_items" not in plan:
        pytest.skip("no request brings enough rows")
    items = _items(plan)
    units = len(items) * Hkv
    parts, rows, n = plan["tc0_info"]
    sched = plan["tc0_sched"]
    assert rows == ops.TC_ROWS and n == min(units, ctas)
    assert sched[0] == n + 1 and sched[n] == len(sched) == n + 1 + units
    assert all(sched[c] <= sched[c + 1] for c in range(n))
    assert sorted(sched[n + 1:]) == list(range(units))

    def cost(unit):
        req, q0, lo, hi, part = items[unit // Hkv][:5]
        return -(-(hi - lo // ops.TC_BN * ops.TC_BN) // ops.TC_BN) + ops.TC_ITEM_COST_STEPS + (ops.TC_PART_COST_STEPS if part >= 0 else 0)
    loads = [sum(cost(u) for u in sched[sched[c]:sched[c + 1]]) for c in range(n)]
    assert min(loads) > 0, "with as many CTAs as units at most, every CTA has work"
    # longest first to the least loaded: no CTA carries more than the lightest one plus one unit
    assert max(loads) - min(loads) <= max(cost(u) for u in range(units)) + 1e-3
    again = ops.plan_attention(q_lens, ctx_lens, 16, ((Hq, Hkv, D, window),), torch.bfloat16)
    assert again["tc0_sched"] == sched and again["tc0_items"] == plan["tc0_items"]


def test_long_tiles_are_cut_only_where_the_schedule_gains():
    geo = ((16, 8, 128, 0),)
    one = ops.plan_attention([2048], [0], 16, geo, torch.bfloat16)
    assert 0 < one["tc0_info"][0] <= 16, "a single long prompt: its longest tiles are cut, in few parts"
    many = ops.plan_attention([1024] * 16, [0] * 16, 16, geo, torch.bfloat16)
    assert many["tc0_info"][0] == 0, "enough tiles for every SM: nothing is cut"
    behind = ops.plan_attention([128], [30000], 16, geo, torch.bfloat16)
    assert behind["tc0_info"][0] >= 2, "one tile behind a long context is cut so that more than 8 SMs work"


@pytest.mark.parametrize("seed", range(8))
def test_parts_by_length_cover_every_key_in_a_fixed_number_of_items(seed):
    """Decoded tokens whose contexts are cut by their lengths: the lists' lengths and the scratch depend on the total alone, every
    request has the parts it was given, longest first, and what is left over are items without rows."""
    rng = random.Random(200 + seed)
    geo = ((16, 8, 128, 0), (32, 8, 128, 0), (16, 8, 128, 700, True), (16, 8, 128, 0, False, 3))[seed % 4]
    R = rng.randint(10, 18)
    ctx = [rng.choice([0, 1, 200, 255, 256, 3000, 9000, rng.randint(1, 2000)]) for _ in range(R)]
    total = ops.TotalParts(rng.choice([R, R + 1, 37, 74]))
    plan = ops.plan_attention([1] * R, ctx, 16, (geo,), torch.bfloat16, uniform_splits={geo: total})
    items = _items(plan, "fa0_items")
    assert len(items) == total and plan["fa0_info"] == [total, geo[0] // geo[1], 1, geo[0] // geo[1], 0] and plan["fa0_merge"] == []
    of = {r: [i for i in items if i[8] and i[0] == r] for r in range(R)}
    parts = ops.parts_by_length(ops.attended_keys([1] * R, ctx, geo[3]), total)
    used = [i[4] for i in items if i[4] >= 0]
    assert len(set(used)) == len(used) and max(used, default=0) < total
    for r, mine in of.items():
        assert len(mine) == parts[r] and all(i[7] == r and i[9] == ctx[r] for i in mine)
        if len(mine) == 1:
            assert mine[0][2:7] == [0, ctx[r] + 1, -1, 0, 0]
        else:
            mine.sort(key=lambda i: i[6])
            assert [i[4:7] for i in mine] == [[mine[0][4] + s, len(mine), s] for s in range(len(mine))]
            # the keys of a part as the kernel works them out: equal shares rounded up to its groups of 16 keys, from the first key
            # tile that the window reaches on; together they are every key that the token attends to, each once
            lo = max(0, ctx[r] - geo[3] + 1) // ops.FLASH_BN * ops.FLASH_BN if geo[3] else 0
            per = -(-(-(-(ctx[r] + 1 - lo) // len(mine))) // 16) * 16
            spans = [(lo + s * per, min(ctx[r] + 1, lo + (s + 1) * per)) for s in range(len(mine))]
            keys = [k for a, b in spans for k in range(a, b)]
            assert keys == list(range(lo, ctx[r] + 1)) and keys[0] <= max(0, ctx[r] - geo[3] + 1 if geo[3] else 0)
    empty = [i for i in items if not i[8]]
    assert len(empty) == total - sum(parts) and all(i == [0, 0, 0, 0, -1] + [0] * 7 for i in empty)


def test_contexts_are_cut_by_length_only_where_they_are_unequal():
    geo, bf = (16, 8, 128, 0), torch.bfloat16
    even, ragged = [1000] * 28, [150 + 70 * i for i in range(28)]
    splits = lambda ctx, dtype=bf, g=geo: ops.decode_splits(len(ctx), 2048, (g,), dtype, ctx)[g]
    assert type(splits(ragged)) is ops.TotalParts and splits(ragged) == 37
    assert splits(even) == 1 and type(splits(even)) is int
    assert splits(ragged[:4]) > 1 and type(splits(ragged[:4])) is int, "few requests are cut into clusters"
    assert type(splits(ragged, torch.float32)) is int and type(splits(ragged, g=(16, 8, 64, 0))) is int
    assert type(splits([100 + 10 * i for i in range(28)])) is int, "short contexts stay whole"
    assert splits(ragged * 2 + ragged[:8]) == 74 and type(splits(ragged * 3)) is int
    beside = ops.plan_attention([512] + [1] * 15, [0] + [150 + 130 * i for i in range(15)], 16, (geo,), bf)
    assert len(_items(beside, "fa0_items")) == beside["fa0_info"][0] == 37


def test_latent_attention_shares_an_sm_with_no_other_tensor_memory():
    """Its CTAs take all 512 columns of tensor memory, for which a CTA waits without a limit; a product behind it that held some on
    the same SM would itself wait for this kernel's end.  Whatever the cache row's size, a launch asks for so much shared memory
    that the smallest of those kernels (60 KB) does not fit beside it in an SM's 228 KB, 1 KB of which goes with each CTA."""
    import ctypes
    for D in range(16, 257, 16):
        alone = ctypes.c_int()
        smem = int(ops.lib().qe_latent_attention_tc_smem(D, ctypes.byref(alone)))
        assert alone.value <= smem <= 225 * 1024
        assert smem + 1024 + 60 * 1024 + 1024 > 228 * 1024, D


def test_contexts_are_dealt_out_once_and_not_at_all_where_sums_tell(monkeypatch):
    """A decode step's plan is on the host's path: a batch of equal or nearly equal contexts is told by its sum and by counting the
    parts that it would need, and one that is cut by length is dealt out once, not by ``decode_splits`` and by the plan again."""
    geo, bf = (16, 8, 128, 0), torch.bfloat16
    calls = []
    real = ops.parts_by_length
    monkeypatch.setattr(ops, "parts_by_length", lambda *a: calls.append(1) or real(*a))

    def step(ctx):
        calls.clear()
        splits = ops.decode_splits(len(ctx), 2048, (geo,), bf, ctx)
        ops.plan_attention([1] * len(ctx), ctx, 16, (geo,), bf, uniform_splits=splits)
        return splits[geo]
    for R in (15, 28, 36, 48, 64, 73):
        assert step([1000] * R) == 1 and not calls
        assert step([960 + 16 * (i % 6) for i in range(R)]) == 1 and not calls
    for ragged in ([150 + 70 * i for i in range(28)], [150 + 130 * i for i in range(15)], [120 + 28 * i for i in range(64)]):
        assert type(step(ragged)) is ops.TotalParts and len(calls) == 1
    calls.clear()
    ops.plan_attention([512] + [1] * 15, [0] + [150 + 130 * i for i in range(15)], 16, (geo,), bf)
    assert len(calls) == 1


@pytest.mark.parametrize("seed", range(12))
def test_a_step_of_decoded_tokens_alone_is_planned_as_the_general_path_does(seed):
    """The same requests beside one that brings two tokens take the general path: whole contexts, equal parts, parts by length."""
    rng = random.Random(400 + seed)
    geo = ((16, 8, 128, 0), (32, 8, 128, 0), (16, 8, 128, 700, True), (6, 2, 48, 0))[seed % 4]
    R = rng.randint(1, 40)
    ctx = [rng.choice([0, 255, 256, 1000, rng.randint(1, 5000)]) for _ in range(R)]
    for parts in (1, 2, 3, 8, ops.TotalParts(2 * R)):
        one, both = parts, parts
        if isinstance(parts, ops.TotalParts):
            both = ops.TotalParts(parts + 1)
            both.shares = ops.parts_by_length(ops.attended_keys([1] * R, ctx, geo[3]), parts) + [1]
        got = ops.plan_attention([1] * R, ctx, 16, (geo,), torch.bfloat16, uniform_splits={geo: one})
        want = ops.plan_attention([1] * R + [2], ctx + [0], 16, (geo,), torch.bfloat16, uniform_splits={geo: both})
        rows = lambda plan, key, n: [plan[key][i:i + n] for i in range(0, len(plan[key]), n)]
        held = lambda items: [i for i in items if i[8]]                 # (the items that are left over have no tokens)
        assert held(rows(got, "fa0_items", 12)) == [i for i in held(rows(want, "fa0_items", 12)) if i[0] != R]
        assert rows(got, "fa0_merge", 4) == [m for m in rows(want, "fa0_merge", 4) if m[0] != R]
        assert len(got["fa0_items"]) // 12 == (parts if isinstance(parts, ops.TotalParts) else parts * R)
        assert got["tiles"] == want["tiles"][:-2]
        G = geo[0] // geo[1]
        n_parts = int(parts) if isinstance(parts, ops.TotalParts) else parts * R if parts > 1 else 0
        assert got["fa0_info"] == [n_parts, G if n_parts else 1, 1, G, parts if parts in (2, 8) and not isinstance(parts, ops.TotalParts) else 0]


@pytest.mark.parametrize("heads,kv_heads,ctx", [
    (16, 8, [800 + 11 * i for i in range(37)]),             # one round of whole contexts: 29.0 us whole, 34.6 cut
    (32, 8, [800 + 11 * i for i in range(37)]),             # 29.7, 38.9
    (32, 8, [130 + 42 * i for i in range(39)]),             # 26.9, 31.7
    (32, 8, [175 + 1225 * (i % 2) for i in range(48)]),     # 39.3, 42.4
    (32, 4, [560 + 4 * i for i in range(74)]),              # 21.8, 38.0
    (16, 1, [560 + i for i in range(296)]),                 # 25.2, 52.2
    (64, 8, [1000] * 10),                                   # eight rows an item: 14.6, 18.0
    (64, 8, [150] * 10 + [900] * 3),                        # 12.0, 15.8
    (32, 8, [1000] * 12),                                   # 14.6, 15.7
])
def test_contexts_stay_whole_where_cutting_them_costs_more(heads, kv_heads, ctx):
    geo, bf = (heads, kv_heads, 128, 0), torch.bfloat16
    splits = ops.decode_splits(len(ctx), -(-max(ctx) // 1024) * 1024, (geo,), bf, ctx)[geo]
    assert type(splits) is int
    beside = ops.plan_attention([512] + [1] * len(ctx), [0] + ctx, 16, (geo,), bf)
    whole = ops.FLASH_TARGET_CTAS // (len(ctx) * kv_heads) <= 1
    assert not whole or beside["fa0_info"][0] == 0


@pytest.mark.parametrize("heads,kv_heads,ctx", [
    (16, 8, [150 + 70 * i for i in range(28)]), (64, 8, [200] * 16 + [4000]), (32, 8, [150 + 130 * i for i in range(15)]),
    (16, 8, [200] * 36 + [8192]), (32, 8, [350] * 55 + [3500]), (16, 4, [150 + 50 * i for i in range(111)]), (16, 1, [200] * 99 + [8192]),
])
def test_contexts_are_cut_where_one_of_them_sets_the_time(heads, kv_heads, ctx):
    geo, bf = (heads, kv_heads, 128, 0), torch.bfloat16
    assert type(ops.decode_splits(len(ctx), -(-max(ctx) // 1024) * 1024, (geo,), bf, ctx)[geo]) is ops.TotalParts


@pytest.mark.parametrize("heads,kv_heads,q_lens,ctx_lens,want", [
    (16, 8, [2], [600], 4), (16, 8, [2], [1100], 8), (16, 8, [4], [1700], 4), (16, 8, [8], [1200], 4), (8, 8, [2], [1400], 8),     # 3, 5, 7 splits of
    (16, 8, [2, 2], [700, 700], 4), (16, 8, [2], [3000], 8), (16, 2, [2] * 18, [1300] * 18, 2), (16, 8, [2] * 8, [330] * 8, 2),    # 256 keys: the next cluster
    (16, 8, [2] * 10, [700] * 10, 1), (32, 8, [2] * 18, [2900] * 18, 1), (16, 8, [3], [200], 1),
    (16, 8, [2] + [1] * 9, [16000] + [200] * 9, [9] + [1] * 9), (16, 8, [2] + [1] * 5, [16000] + [200] * 5, [13] + [1] * 5),
    (16, 8, [1, 2, 1], [40, 3000, 700], [9, 2]), (16, 8, [2] * 5, [4000] * 5, [4, 4, 4, 3, 3]),
])
def test_a_few_tokens_of_every_request_are_cut_by_their_lengths(heads, kv_heads, q_lens, ctx_lens, want):
    """Contexts of about equal lengths form clusters of exactly 2, 4 or 8 parts, whatever the number of splits; others have parts by
    their lengths, as many CTAs of 8 warps as SMs in all."""
    plan = ops.plan_attention(q_lens, ctx_lens, 16, ((heads, kv_heads, 128, 0),), torch.bfloat16)
    info = plan["fa0_info"]
    if isinstance(want, int):
        assert info[4] == (want if want > 1 else 0) and info[0] == (want * len(q_lens) if want > 1 else 0)
        return
    parts = {i[0]: i[5] or 1 for i in _items(plan, "fa0_items")}
    assert info[4] == 0 and info[0] == len(plan["fa0_items"]) // 12 <= ops.TC_TARGET_CTAS // kv_heads and plan["fa0_merge"] == []
    assert sorted((n for n in parts.values()), reverse=True)[:len(want)] == want


@pytest.mark.parametrize("seed", range(24))
def test_a_few_tokens_of_every_request_leave_no_key_and_no_place_out(seed):
    """Any batch of a few tokens of every request: each request's parts are there once, with places of their own in the scratch
    memory, which holds no more than an item of every CTA."""
    rng = random.Random(600 + seed)
    geo = ((16, 8, 128, 0), (32, 8, 128, 0), (16, 2, 128, 700), (8, 8, 128, 0, True), (16, 4, 128, 0, False, 3), (40, 40, 128, 0))[seed % 6]
    G, R = geo[0] // geo[1], rng.randint(1, 20)
    q = [rng.choice([1, rng.randint(1, 16 // G)]) for _ in range(R)]
    q[rng.randrange(R)] = rng.randint(2, 16 // G)
    ctx = [rng.choice([0, 40, 256, rng.randint(1, 2000), rng.randint(1, 20000) if rng.random() < 0.2 else 500]) for _ in range(R)]
    plan = ops.plan_attention(q, ctx, 16, (geo,), torch.bfloat16)
    items, (n_parts, part_rows, small, most, same) = _items(plan, "fa0_items"), plan["fa0_info"]
    held = [i for i in items if i[8]]
    assert small == 1 and most == max(q) * G and (not n_parts or part_rows >= max(n for i, n in enumerate(q) if any(h[0] == i and h[4] >= 0 for h in held)) * G)
    places = [i[4] for i in held if i[4] >= 0]
    assert sorted(places) == sorted(set(places)) and max(places, default=-1) < max(1, n_parts)
    for r in range(R):
        mine = sorted((i for i in held if i[0] == r), key=lambda i: i[6])
        assert all(i[7:10] == [sum(q[:r]), q[r], ctx[r]] for i in mine)
        if len(mine) == 1 and mine[0][4] < 0:
            assert mine[0][2:7] == [0, ctx[r] + q[r], -1, 0, 0]
        else:
            assert [i[4:7] for i in mine] == [[mine[0][4] + s, len(mine), s] for s in range(len(mine))]
            assert not same or len(mine) == same
    if same:
        assert same in (2, 4, 8) and len(items) == n_parts == same * R and [i[0] for i in items] == [r for r in range(R) for _ in range(same)]
