"""Host arithmetic of the decode schedule (the kernel computes the same split on the device)."""
import numpy as np
import pytest

from hy3_b200.attn import decode_schedule, prefill_schedule


@pytest.mark.parametrize("lens,heads,ctas", [([32768], 8, 148), ([1], 8, 148), ([128, 129, 0, 5000], 8, 148),
                                              ([1000] * 64, 4, 148), ([65536, 1024], 1, 7), ([0, 0], 8, 148),
                                              ([300] * 18, 8, 148), ([300] * 19, 8, 148), ([70000, 5], 8, 148),
                                              ([1024 + (7919 * i) % 64513 for i in range(64)], 1, 148), ([5000] * 16, 8, 148)])
def test_schedule_partitions_units(lens, heads, ctas):
    """Every unit belongs to exactly one CTA; ranges are ordered; with few segments no range crosses a
    segment boundary; with many segments the ranges are balanced to one page."""
    pages = [(n + 127) // 128 for n in lens]
    total = sum(pages) * heads
    ranges = []
    for c in range(ctas):
        tot, u0, u1 = decode_schedule(lens, heads, ctas, c)
        assert tot == total and u1 >= u0
        if u1 > u0:
            ranges.append((u0, u1))
    assert sorted(ranges) == ranges
    covered = 0
    for u0, u1 in ranges:
        assert u0 == covered
        covered = u1
    assert covered == total
    sizes = [b - a for a, b in ranges]
    if len(lens) * heads < ctas and ranges and max(sizes) - min(sizes) > 1:
        # the aligned split (whole CTAs per segment) was kept: nobody has more than 5/4 of the even share (+ 1 page)
        assert max(sizes) * 4 <= -(-total // ctas) * 5 + 4
        bounds = set()
        acc = 0
        for p in pages:
            for _ in range(heads):
                bounds.add(acc)
                acc += p
        for u0, u1 in ranges:
            assert not any(u0 < b < u1 for b in bounds), "a CTA straddles two segments"
    elif ranges and len(lens) * heads >= ctas:
        assert max(sizes) - min(sizes) <= 1


def test_piece_count_formula_matches_ranges():
    """c_first / c_last as computed in the kernel: ceil((u+1)*C/U)-1 is the CTA that owns unit u."""
    rng = np.random.default_rng(0)
    for _ in range(200):
        C = int(rng.integers(1, 300))
        U = int(rng.integers(1, 5000))
        starts = [c * U // C for c in range(C + 1)]
        for u in rng.integers(0, U, 20):
            u = int(u)
            owner = -(-((u + 1) * C) // U) - 1
            assert starts[owner] <= u < starts[owner + 1]


def test_plan_eval_follows_the_reference_walk():
    """hy3_gpu.cu:857-889: with a chunk size and more than one token, all tokens but the last go through chunks; the
    position of the first token is cache_len / n_layers."""
    from hy3_b200.session import plan_eval, read_env
    assert plan_eval(0, 3, 80, 0) == [("token", 0), ("token", 1), ("token", 2)]
    assert plan_eval(160, 1300, 80, 512) == [("chunk", 2, 512), ("chunk", 514, 512), ("chunk", 1026, 275), ("token", 1301)]
    assert plan_eval(80, 1, 80, 512) == [("token", 1)]                     # a single token never takes the chunk path
    assert plan_eval(0, 2, 80, 512) == [("chunk", 0, 1), ("token", 1)]
    assert plan_eval(0, 513, 2, 512) == [("chunk", 0, 512), ("token", 512)]
    e = read_env({"HY3_KV_INT4": "1", "HY3_PREFILL_CHUNK": "abc", "HY3_POS_STRIDE": "-3", "HY3_POS_JUMP": "7"})
    assert e == {"kv_dtype": "int4", "chunk": 0, "pos_stride": 1, "pos_jump": 7, "pos_jump_at": 0}
    assert read_env({})["kv_dtype"] == "int8" and read_env({"HY3_KV_FP16": "1"})["kv_dtype"] == "fp16"


@pytest.mark.parametrize("base,nq", [(0, 1), (0, 32), (0, 33), (1001, 45), (5, 59), (31, 64), (4096, 512), (0, 2048), (2048, 953), (16000, 128),
                                     (262143, 1), (262000, 2048), (1000, 1000), (0, 8192), (100, 8193), (4194304, 7)])
@pytest.mark.parametrize("heads", [8, 4, 3, 1])
@pytest.mark.parametrize("records", [512, 16, 0])
def test_prefill_schedule_covers_every_step_once(base, nq, heads, records):
    """The pieces of a block are its steps [0, n) without gap or overlap, the records of cut blocks are disjoint and within the
    scratch, and the table is in descending order of length."""
    t = prefill_schedule(base, nq, heads, 148, records)
    nqb = -(-nq // 32)
    if len(t) == 0:      # uncut
        assert records < 512 or (base, nq, heads) != (16000, 128, 8)
        return
    assert (np.diff(t[:, 2]) <= 0).all() and (t[:, 2] >= 1).all()
    used = np.zeros(records // heads + 1, int)
    for b in range(nqb):
        p = t[t[:, 0] == b]
        p = p[np.argsort(p[:, 4])]
        assert (p[:, 5] == len(p)).all() and (p[:, 4] == np.arange(len(p))).all()
        assert (p[:, 1] == np.concatenate([[0], np.cumsum(p[:-1, 2])])).all()
        assert p[:, 2].sum() == -(-min(base + 32 * b + 32, base + nq) // 64)
        if len(p) > 1:
            assert (p[:, 3] == p[0, 3]).all() and (p[0, 3] + len(p)) * heads <= records
            used[p[0, 3]:p[0, 3] + len(p)] += 1
    assert used.max() <= 1 and len(t) == sum((t[:, 0] == b).sum() for b in range(nqb))


def _few_row_batches():
    rng = np.random.default_rng(17)
    out = [([262144] + [100] * 4, 8), ([262144] + [128] * 31, 2), ([0, 5, 0, 9000, 0, 7, 3, 1], 8), ([1] * 18, 8), ([4096] * 17, 8), ([0] * 6, 8)]
    for n in (2, 3, 5, 8, 17, 18, 31, 32, 33, 40):
        for heads in (8, 5, 4, 3, 2, 1):
            for hi in (300, 3000, 60000):
                lens = rng.integers(1, hi, n)
                lens[rng.random(n) < 0.15] = 0
                if rng.random() < 0.3:
                    lens[int(rng.integers(n))] = 20 * hi
                out.append(([int(x) for x in lens], heads))
    return out


@pytest.mark.parametrize("dt", ["int4", "fp16", "int8"])
def test_schedule_of_few_rows(dt):
    """Ragged batches around the 2 to 32 rows that the FP16 / INT4 kernel cuts into pieces of even size: every page of every segment
    in exactly one CTA, ranges in order; either no CTA straddles two segments, and then no piece is far above the even share, or the
    ranges are equal."""
    ctas, even_seen = 148, 0
    for lens, heads in _few_row_batches():
        pages = [-(-n // 128) for n in lens]
        total = sum(pages) * heads
        got = [decode_schedule(lens, heads, ctas, c, kv_dtype=dt) for c in range(ctas)]
        assert all(g[0] == total for g in got)
        r = [(u0, u1) for _, u0, u1 in got if u1 > u0]
        assert [u0 for u0, _ in r] == [0] * bool(r) + [u1 for _, u1 in r[:-1]] and (r[-1][1] if r else 0) == total
        if not r:
            continue
        sizes = [b - a for a, b in r]
        bounds = np.cumsum([p for p in pages for _ in range(heads)])
        straddles = any(((bounds > a) & (bounds < b)).any() for a, b in r)
        even, segs = -(-total // ctas), len(lens) * heads
        if straddles:
            assert max(sizes) - min(sizes) <= 1
        elif dt != "int8" and 2 <= len(lens) <= 32 and segs < ctas < 4 * segs:
            even_seen += max(sizes) - min(sizes) > 1
            assert max(sizes) * 4 <= even * 5 + 4 or max(sizes) <= even + 5
        elif segs < ctas < 4 * segs and max(sizes) - min(sizes) > 1:
            assert max(sizes) * 4 <= even * 5 + 4
    assert (even_seen >= 10) == (dt != "int8")      # the batches above do reach the even pieces


def test_schedule_depends_on_the_cache_type():
    """8 rows of 22 to 56 pages x 8 heads on 148 CTAs: whole CTAs per segment with at most 19 pages each (FP16 / INT4), or equal ranges
    (INT8); and the shortened last pieces of an INT8 single-row grid."""
    lens = [3006, 7075, 3290, 3374, 6828, 2718, 2910, 3288]
    for dt, worst in (("int4", 19), ("fp16", 19), ("int8", 14)):
        r = [decode_schedule(lens, 8, 148, c, kv_dtype=dt)[1:] for c in range(148)]
        assert max(b - a for a, b in r) == worst, dt
    one = {dt: [b - a for _, a, b in (decode_schedule([32768], 8, 148, c, kv_dtype=dt) for c in range(126, 144))] for dt in ("int8", "int4")}
    assert sum(one["int8"]) == sum(one["int4"]) == 256 and min(one["int4"]) == 14
    assert one["int8"][-4:] == [13, 12, 13, 13] and min(one["int8"][:-4]) >= 14, one


@pytest.mark.parametrize("dt", ["int4", "fp16"])
def test_even_pieces_are_the_least_that_fit(dt):
    """The piece size is the least for which the pieces fit the grid, also with one very long row among short ones, and a split that
    the rule accepts is not lost."""
    rng = np.random.default_rng(23)
    batches = _few_row_batches()
    for n, heads in ((5, 8), (10, 4), (20, 2), (32, 2), (18, 8)):
        for long_pages in (500, 2048, 8192):
            batches.append(([128 * long_pages] + [128] * (n - 1), heads))
            batches.append(([128 * int(x) for x in rng.integers(1, 40, n - 1)] + [128 * long_pages], heads))
    seen = 0
    for lens, heads in batches:
        n, P = len(lens), [-(-x // 128) for x in lens]
        if not (2 <= n <= 32 and n * heads < 148 < 4 * n * heads) or sum(P) == 0:
            continue
        cap, even = 148 // heads, -(-sum(P) * heads // 148)
        least = next(L for L in range(-(-sum(P) // cap), max(P) + 1) if sum(-(-p // L) for p in P) <= cap)
        r = [decode_schedule(lens, heads, 148, c, kv_dtype=dt)[1:] for c in range(148)]
        sizes = [b - a for a, b in r if b > a]
        if least * 4 <= even * 5 + 4 or least <= even + 5:
            assert max(sizes) <= least and len(sizes) == heads * sum(-(-p // least) for p in P), (lens, heads)
            seen += 1
        else:
            assert max(sizes) - min(sizes) <= 1
    assert seen > 20


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("length,heads", [(128 * 24, 1), (128 * 25, 1), (20000, 1), (60000, 2), (33000, 4), (32768, 8), (1 << 20, 1), (1 << 20, 8)])
def test_schedule_bounds_the_pieces_of_a_segment(dt, length, heads):
    """A segment of p pages is cut into at most 24 + p / 32 pieces, evenly, and every page belongs to one of them."""
    p = -(-length // 128)
    ranges = [r for r in (decode_schedule([length], heads, 148, c, dt)[1:] for c in range(148)) if r[1] > r[0]]
    assert len(ranges) == heads * min(1 + (148 - heads) // heads, 24 + p // 32, p)
    assert ranges[0][0] == 0 and ranges[-1][1] == p * heads and all(a[1] == b[0] for a, b in zip(ranges, ranges[1:]))
    sizes = [b - a for a, b in ranges]
    assert max(sizes) - min(sizes) <= (1 if dt != "int8" else 4)      # INT8: the pieces that start late take two pages less
