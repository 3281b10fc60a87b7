"""GPU parity of the split-KV GQA decode kernel (and its LSE-merge epilogue) through the C ABI,
against the oracle attention (restatement of hy3.c:617-652) evaluated on the same stored K/V."""
import numpy as np
import pytest

from helpers import SEED, check_attention, make_slots, slots_to_float

pytestmark = pytest.mark.gpu

LENS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1000, 4097]


def load_cache(ctx, oracle, dt, layer, seq, K, V):
    ks, vs = make_slots(oracle, K, dt), make_slots(oracle, V, dt)
    ctx.import_kv(layer, seq, 0, ks, vs)
    return slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)


@pytest.fixture(params=["staged", "direct"])
def variant(request, monkeypatch):
    """The two load paths of the decode kernel: bulk-copy ring in shared memory, or direct 128-bit loads."""
    monkeypatch.delenv("HY3A_DECODE_STAGES", raising=False)
    if request.param == "direct":
        monkeypatch.setenv("HY3A_DECODE_STAGES", "0")
    return request.param


@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_decode_lengths(cuda, oracle, dt, variant):
    import torch
    from hy3_b200 import Hy3Attn
    nmax = max(LENS)
    ctx = Hy3Attn(kv_dtype=dt, n_layers=3, max_batch=4, max_tokens=nmax + 256)
    K = oracle.fill_normal((nmax, 8, 128), SEED, 51)
    V = oracle.fill_normal((nmax, 8, 128), SEED, 52)
    Kf, Vf = load_cache(ctx, oracle, dt, 2, 0, K, V)
    ks, vs = ctx.export_kv(2, 0, 0, nmax)          # import/export round trip is the identity
    assert np.array_equal(ks, make_slots(oracle, K, dt)) and np.array_equal(vs, make_slots(oracle, V, dt))
    q = oracle.fill_normal((64, 128), SEED, 53)
    tq = torch.from_numpy(q[None]).to(cuda)
    worst = 0.0
    for n in LENS:
        ctx.batch_set([0], [n - 1])
        out = ctx.decode(2, tq)
        ctx.sync()
        err, _ = check_attention(out[0].cpu().numpy(), oracle.attention(q, Kf[:n], Vf[:n]), "%s ntok=%d" % (dt, n))
        worst = max(worst, err)
    print("decode %s worst max-abs vs oracle-on-stored-KV: %.3g" % (dt, worst))
    ctx.close()


@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_decode_long_context_many_ctas(cuda, oracle, dt, variant):
    """Long enough that every CTA gets work and (row, head) segments span many CTAs (merge epilogue)."""
    import torch
    from hy3_b200 import Hy3Attn
    n = 40000
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=2, max_tokens=n + 128)
    K = oracle.fill_normal((n, 8, 128), SEED, 61)
    V = oracle.fill_normal((n, 8, 128), SEED, 62)
    Kf, Vf = load_cache(ctx, oracle, dt, 0, 0, K, V)
    q = 1.5 * oracle.fill_normal((64, 128), SEED, 63)
    tq = torch.from_numpy(q[None]).to(cuda)
    ctx.batch_set([0], [n - 1])
    for _ in range(3):                              # repeated launches reuse the self-resetting counters
        out = ctx.decode(0, tq)
    ctx.sync()
    want = oracle.attention_f64(q, Kf, Vf).astype(np.float32)
    check_attention(out[0].cpu().numpy(), want, "%s ntok=%d" % (dt, n))
    ctx.close()


@pytest.mark.parametrize("dt", ["fp16", "int4", "int8"])
def test_decode_is_bitwise_repeatable(cuda, dt):
    """The same launch repeated back to back gives the same bits: fold orders are fixed, and no warp may read a ring stage
    that is still being filled (FP16 pages leave room for a two-stage ring only; a consumer warp that holds no granule of
    a page used to be able to pass its next wait on a stale barrier phase there)."""
    import torch
    from hy3_b200 import Hy3Attn
    n = 40000
    ctx = Hy3Attn(kv_dtype=dt, n_layers=2, max_batch=2, max_tokens=n + 128)
    for l in range(2):
        ctx.fill_random(l, 0, 0, n, 3 + l)
    q = torch.randn((1, 64, 128), device=cuda, generator=torch.Generator(device=cuda).manual_seed(5))
    ctx.batch_set([0], [n - 1])
    ref = [ctx.decode(l, q).clone() for l in range(2)]
    torch.cuda.synchronize()
    differing = 0
    for _ in range(60):
        outs = [(l, ctx.decode(l, q)) for _ in range(3) for l in range(2)]
        torch.cuda.synchronize()
        differing += sum(0 if torch.equal(o, ref[l]) else 1 for l, o in outs)
    ctx.sync()
    ctx.close()
    assert differing == 0, "%d of 360 launches differ from the first" % differing


@pytest.mark.parametrize("dt", ["int4", "fp16"])
@pytest.mark.parametrize("n", [40017, 351])
def test_ring_depth_does_not_matter(cuda, dt, n, monkeypatch):
    """Every depth of the page ring gives the same bits, back to back (a consumer warp skips pages: up to two INT4 pages lie
    between its 32-token granules), and 32-token granules end anywhere in the last page."""
    import torch
    from hy3_b200 import Hy3Attn
    q = torch.randn((1, 64, 128), device=cuda, generator=torch.Generator(device=cuda).manual_seed(6))
    ref = None
    for stages in (None, 2) if dt == "fp16" else (None, 2, 3, 5, 7):
        if stages is None:
            monkeypatch.delenv("HY3A_DECODE_STAGES", raising=False)
        else:
            monkeypatch.setenv("HY3A_DECODE_STAGES", str(stages))
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=1, max_tokens=n + 128)
        ctx.fill_random(0, 0, 0, n, 9)
        outs = []
        for m in (n, n - 1, n - 15, n - 16, n - 17, n - 31, n - 32, n - 33):
            ctx.batch_set([0], [m - 1])
            outs += [ctx.decode(0, q).clone() for _ in range(8)]
        ctx.sync()
        ctx.close()
        ref = ref or outs
        assert all(torch.equal(a, b) for a, b in zip(outs, ref)), "stages=%s" % stages
        assert all(torch.equal(outs[i], outs[i - i % 8]) for i in range(len(outs)))


@pytest.mark.parametrize("lens", [[40017], [351], [351, 65, 700, 129, 1, 64] * 4])
def test_half_page_ring_depth_does_not_matter(cuda, lens, monkeypatch):
    """An FP16 ring holds half pages, 5 of them or as few as 2 (4 beside the largest batches): every depth gives the same bits, back to
    back.  The rows of the batch are more segments than CTAs, and a row that ends in the first half of a page puts the CTA's next
    segment at an odd position of the ring."""
    import torch
    from hy3_b200 import Hy3Attn
    B = len(lens)
    q = torch.randn((B, 64, 128), device=cuda, generator=torch.Generator(device=cuda).manual_seed(7))
    ref = None
    for stages in ("5", "4", "3", "2"):
        monkeypatch.setenv("HY3A_DECODE_STAGES", stages)
        ctx = Hy3Attn(kv_dtype="fp16", n_layers=1, max_seqs=B, max_batch=B, max_tokens=sum(lens) + 128 * B, max_tokens_per_seq=max(lens) + 128)
        for i, n in enumerate(lens):
            ctx.fill_random(0, i, 0, n, 30 + i)
        outs = []
        for cut in (1, 2, 33, 64, 65):
            ctx.batch_set(list(range(B)), [max(0, n - cut) for n in lens])
            outs += [ctx.decode(0, q).clone() for _ in range(8)]
        ctx.sync()
        ctx.close()
        ref = ref or outs
        assert all(torch.equal(a, b) for a, b in zip(outs, ref)), "stages=%s" % stages
        assert all(torch.equal(outs[i], outs[i - i % 8]) for i in range(len(outs)))


@pytest.mark.parametrize("dt", ["int4", "fp16"])
@pytest.mark.parametrize("heads", [8, 3])
@pytest.mark.parametrize("lens", [[3007, 129, 1, 4097, 640], [300] * 17, [1, 5000, 128, 2, 3, 257, 127, 255, 31, 33, 700, 900, 11]])
def test_few_rows_in_even_pieces(cuda, oracle, dt, heads, lens):
    """2 to 32 rows with fewer than four CTAs per segment: whole CTAs per segment in pieces of even size (or, where that is
    unbalanced, the equal split); every row against the oracle."""
    import torch
    from hy3_b200 import Hy3Attn
    B = len(lens)
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=B, max_batch=B, kv_head_count=heads, max_tokens=sum(lens) + 128 * B, max_tokens_per_seq=8192)
    for i, n in enumerate(lens):
        ctx.fill_random(0, i, 0, n, 70 + i)
    q = oracle.fill_normal((B, 64, 128), SEED, 441)
    ctx.batch_set(list(range(B)), [n - 1 for n in lens])
    out = ctx.decode(0, torch.from_numpy(q).to(cuda))
    ctx.sync()
    out = out.cpu().numpy()
    for i, n in enumerate(lens):
        ks, vs = ctx.export_kv(0, i, 0, n)
        Kf, Vf = slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)
        want = oracle.attention(q[i], Kf, Vf)
        check_attention(out[i][:8 * heads], want[:8 * heads], "%s row %d len %d" % (dt, i, n))
    ctx.close()


@pytest.mark.parametrize("dt,stages", [("int8", None), ("int4", None), ("fp16", None), ("int4", 2)])
@pytest.mark.parametrize("lens", [[32700], [36800], [66000], [9000] * 40])
def test_folds_of_many_records(cuda, oracle, dt, stages, lens, monkeypatch):
    """One KV head: 32, 33 and 40 pieces of a segment (one record per lane of the folding warp, one more, and several landings in a ring
    of two pages), and rows whose few pieces straddle CTAs; twice, because every fold leaves its counters for the next launch."""
    import torch
    from hy3_b200 import Hy3Attn
    if stages:
        monkeypatch.setenv("HY3A_DECODE_STAGES", str(stages))
    B = len(lens)
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=B, max_batch=B, kv_head_count=1, max_tokens=sum(lens) + 128 * B, max_tokens_per_seq=max(lens) + 128)
    for i, n in enumerate(lens):
        ctx.fill_random(0, i, 0, n, 170 + i)
    q = oracle.fill_normal((B, 64, 128), SEED, 443)
    ctx.batch_set(list(range(B)), [n - 1 for n in lens])
    outs = [ctx.decode(0, torch.from_numpy(q).to(cuda))[:, :8].clone() for _ in range(2)]
    ctx.sync()
    assert torch.equal(outs[0], outs[1])
    out = outs[0].cpu().numpy()
    for i in sorted({0, B // 3, B - 1}):
        ks, vs = ctx.export_kv(0, i, 0, lens[i])
        want = oracle.attention(q[i], slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt))
        check_attention(out[i], want[:8], "%s row %d of %d" % (dt, i, B))
    ctx.close()


@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
@pytest.mark.parametrize("lens,heads", [([30000] + [100] * 198, 1), ([40000] + [200] * 30, 8)])
def test_folds_of_straddling_segments(cuda, oracle, dt, lens, heads):
    """Equal ranges of units: the pieces of a segment that straddles CTAs meet in the few places that the ring leaves (11; INT8: 3), in
    several landings, while the other warps of the CTA go on to its next segment.  Every lane of the folding warp reads records that
    only one lane has waited for: back to back, bit for bit, and against the oracle."""
    import torch
    from hy3_b200 import Hy3Attn
    from hy3_b200.attn import decode_schedule
    B = len(lens)
    ranges = [decode_schedule(lens, heads, 148, c, kv_dtype=dt)[1:] for c in range(148)]
    first = (lens[0] + 127) // 128                                            # units of row 0's first head
    mine = [r for r in ranges if r[0] < first]
    assert len(mine) > 11 and mine[-1][1] > first                             # many pieces, the last CTA holds the next segment as well
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=B, max_batch=B, kv_head_count=heads, max_tokens=sum(lens) + 128 * B, max_tokens_per_seq=max(lens) + 128)
    for i, n in enumerate(lens):
        ctx.fill_random(0, i, 0, n, 270 + i)
    q = oracle.fill_normal((B, 64, 128), SEED, 445)
    tq = torch.from_numpy(q).to(cuda)
    ctx.batch_set(list(range(B)), [n - 1 for n in lens])
    outs = [ctx.decode(0, tq)[:, :8 * heads].clone() for _ in range(40)]
    ctx.sync()
    assert all(torch.equal(outs[0], o) for o in outs[1:])
    out = outs[0].cpu().numpy()
    for i in (0, 1, 2, B - 1):
        ks, vs = ctx.export_kv(0, i, 0, lens[i])
        want = oracle.attention(q[i], slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt))
        check_attention(out[i], want[:8 * heads], "%s row %d of %d" % (dt, i, B))
    ctx.close()


def test_decode_ragged_batch_and_poison(cuda, oracle):
    """Several sequences of different lengths in one launch; cache bytes past each length are poison."""
    import torch
    from hy3_b200 import Hy3Attn
    lens = [1, 130, 257, 1000, 77, 128, 3000]
    B = len(lens)
    ctx = Hy3Attn(kv_dtype="int8", n_layers=2, max_seqs=B, max_batch=B, max_tokens=sum(lens) + 128 * B, max_tokens_per_seq=4096)
    Kf, Vf = [], []
    for s, n in enumerate(lens):
        cap = (n + 127) // 128 * 128
        K = oracle.fill_normal((cap, 8, 128), SEED, 100 + s)
        V = oracle.fill_normal((cap, 8, 128), SEED, 200 + s)
        K[n:] = 1e4                                  # poison past the valid length (finite, huge)
        V[n:] = -1e4
        a, b = load_cache(ctx, oracle, "int8", 1, s, K, V)
        Kf.append(a[:n]); Vf.append(b[:n])
    q = oracle.fill_normal((B, 64, 128), SEED, 300)
    ctx.batch_set(list(range(B)), [n - 1 for n in lens])
    out = ctx.decode(1, torch.from_numpy(q).to(cuda))
    ctx.sync()
    out = out.cpu().numpy()
    for s in range(B):
        check_attention(out[s], oracle.attention(q[s], Kf[s], Vf[s]), "seq %d len %d" % (s, lens[s]))
    ctx.close()


def test_decode_many_segments_share_ctas(cuda, oracle):
    """More (row, KV head) segments than CTAs: every CTA walks through several segments and segments straddle CTAs
    (the equal-unit-range schedule); a fused step, so that the appends land in many different CTAs."""
    import torch
    from hy3_b200 import Hy3Attn
    rng = np.random.default_rng(7)
    lens0 = [int(x) for x in rng.integers(1, 900, size=40)]      # 320 segments for 148 CTAs
    lens0[3], lens0[17] = 0, 2600
    B = len(lens0)
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_seqs=B, max_batch=B, max_tokens=sum(lens0) + 256 * B, max_tokens_per_seq=4096)
    for s_, n0 in enumerate(lens0):
        if n0:
            ctx.fill_random(0, s_, 0, n0, 500 + s_)
    q = oracle.fill_normal((2, B, 64, 128), SEED, 331)
    k = oracle.fill_normal((2, B, 8, 128), SEED, 332)
    v = oracle.fill_normal((2, B, 8, 128), SEED, 333)
    tq, tk, tv = (torch.from_numpy(x).to(cuda) for x in (q, k, v))
    qo = torch.zeros((B, 64, 128), dtype=torch.float32, device=cuda)
    for t in range(2):
        ctx.batch_set(list(range(B)), [n0 + t for n0 in lens0])
        out = ctx.decode_step(0, tq[t], tk[t], tv[t], q_out=qo)
    ctx.sync()
    out, qo = out.cpu().numpy(), qo.cpu().numpy()
    for s_ in range(B):
        ks, vs = ctx.export_kv(0, s_, 0, lens0[s_] + 2)
        check_attention(out[s_], oracle.attention(qo[s_], slots_to_float(oracle, ks, "int8"), slots_to_float(oracle, vs, "int8")), "seq %d len %d" % (s_, lens0[s_] + 2))
    ctx.close()


def test_append_then_decode_end_to_end(cuda, oracle):
    """The real step: fused append of token t, then attention over [0, t], for a few steps."""
    import torch
    from hy3_b200 import Hy3Attn
    steps, eps = 140, 1e-6
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_batch=1, max_tokens=512, rms_eps=eps)
    w = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    ctx.set_norm_weights(0, w[0], w[1])
    inv, af = oracle.rope_table()
    q = oracle.fill_normal((steps, 64, 128), SEED, 71)
    k = oracle.fill_normal((steps, 8, 128), SEED, 72)
    v = oracle.fill_normal((steps, 8, 128), SEED, 73)
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    outs = []
    for t in range(steps):
        ctx.batch_set([0], [t])
        qo = ctx.append(0, tq[t:t + 1], tk[t:t + 1], tv[t:t + 1])
        outs.append((qo, ctx.decode(0, qo)))
    ctx.sync()
    ks, vs = ctx.export_kv(0, 0, 0, steps)
    Kf, Vf = slots_to_float(oracle, ks, "int8"), slots_to_float(oracle, vs, "int8")
    for t in (0, 1, 15, 16, 127, 128, 139):
        qo, out = outs[t]
        oq, ok = oracle.qk_norm_rope(q[t], k[t], w[0], w[1], eps, t, inv, af)
        # the cache holds exactly what the oracle pipeline would have stored (K within +-1 code of ulp effects)
        want_k = oracle.stored_kv(ok, "int8")
        assert np.abs(Kf[t] - want_k).max() <= 1.01 * np.abs(ok).max() / 127
        check_attention(out[0].cpu().numpy(), oracle.attention(qo[0].cpu().numpy(), Kf[:t + 1], Vf[:t + 1]), "step %d" % t)
        # against the un-quantised fp32 pipeline: report the INT8 bound separately
    t = steps - 1
    oq_all = [oracle.qk_norm_rope(q[i], k[i], w[0], w[1], eps, i, inv, af) for i in range(steps)]
    K32 = np.stack([x[1] for x in oq_all])
    full = oracle.attention(oq_all[t][0], K32, v)
    err = np.abs(outs[t][1][0].cpu().numpy() - full).max()
    print("INT8 KV end-to-end vs un-quantised fp32 pipeline at ntok=%d: max-abs %.3g" % (steps, err))
    assert err < 3e-2
    ctx.close()


@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_fused_step_equals_append_plus_decode(cuda, oracle, dt):
    """hy3a_decode_step (one kernel) against hy3a_append + hy3a_decode: identical cache bytes, identical
    queries, identical outputs; a ragged batch so that page and granule boundaries are crossed."""
    import torch
    from hy3_b200 import Hy3Attn
    lens0 = [0, 15, 16, 127, 128, 300, 2000]          # tokens already cached per sequence
    B, steps = len(lens0), 18
    w = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    q = oracle.fill_normal((steps, B, 64, 128), SEED, 401)
    k = oracle.fill_normal((steps, B, 8, 128), SEED, 402)
    v = oracle.fill_normal((steps, B, 8, 128), SEED, 403)
    res = {}
    for mode in ("two_kernels", "fused"):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=2, max_seqs=B, max_batch=B, max_tokens=4096 + 128 * B, max_tokens_per_seq=2560, rms_eps=1e-6)
        ctx.set_norm_weights(1, w[0], w[1])
        for s_, n0 in enumerate(lens0):
            if n0:
                ctx.fill_random(1, s_, 0, n0, 77)
        outs, qos = [], []
        tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
        for t in range(steps):
            ctx.batch_set(list(range(B)), [n0 + t for n0 in lens0], [n0 + t + 5 for n0 in lens0])
            if mode == "fused":
                qo = torch.zeros((B, 64, 128), dtype=torch.float32, device=cuda)
                out = ctx.decode_step(1, tq[t], tk[t], tv[t], q_out=qo)
            else:
                qo = ctx.append(1, tq[t], tk[t], tv[t])
                out = ctx.decode(1, qo)
            outs.append(out); qos.append(qo)
        ctx.sync()
        caches = [ctx.export_kv(1, s_, 0, n0 + steps) for s_, n0 in enumerate(lens0)]
        res[mode] = (torch.stack(outs).cpu().numpy(), torch.stack(qos).cpu().numpy(), caches)
        if mode == "fused":        # and against the oracle on the stored cache, last step
            for s_ in (0, 3, 6):
                Kf = slots_to_float(oracle, caches[s_][0], dt); Vf = slots_to_float(oracle, caches[s_][1], dt)
                check_attention(res[mode][0][-1, s_], oracle.attention(res[mode][1][-1, s_], Kf, Vf), "fused %s seq %d" % (dt, s_))
        ctx.close()
    a, b = res["two_kernels"], res["fused"]
    assert np.array_equal(a[1], b[1]), "queries differ"
    for (ka, va), (kb, vb) in zip(a[2], b[2]):
        assert np.array_equal(ka, kb) and np.array_equal(va, vb), "cache bytes differ"
    assert np.array_equal(a[0], b[0]), "outputs differ: max %.3g" % np.abs(a[0] - b[0]).max()


def test_partials_and_merge_sequence_shards(cuda, oracle):
    """Two contexts hold the two halves of one sequence; per-shard {m,l,acc} + merge == full attention."""
    import torch
    from hy3_b200 import Hy3Attn
    n, cut = 3000, 1700
    K = oracle.fill_normal((n, 8, 128), SEED, 81)
    V = oracle.fill_normal((n, 8, 128), SEED, 82)
    q = oracle.fill_normal((2, 64, 128), SEED, 83)
    tq = torch.from_numpy(q).to(cuda)
    parts, Kf, Vf = [], [], []
    ctxs = []
    for lo, hi in ((0, cut), (cut, n)):
        ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_seqs=2, max_batch=2, max_tokens=2 * n, max_tokens_per_seq=n + 128)
        a, b = load_cache(ctx, oracle, "int8", 0, 0, K[lo:hi], V[lo:hi])
        Kf.append(a); Vf.append(b)
        ctx.batch_set([0, 1], [hi - lo - 1, -1])     # row 1: a sequence with no keys on this shard
        p = torch.empty((2, 64, 130), dtype=torch.float32, device=cuda)
        ctx.decode(0, tq, partials=p)
        ctx.sync()
        parts.append(p)
        ctxs.append(ctx)
    Kf, Vf = np.concatenate(Kf), np.concatenate(Vf)
    for r, (lo, hi) in enumerate(((0, cut), (cut, n))):
        got = parts[r][0].cpu().numpy()
        want = oracle.attention_partial(q[0], Kf, Vf, lo, hi)
        # same record up to the (m, l, acc) gauge: compare after normalising by the oracle's m
        f = np.exp(got[:, 0] - want[:, 0])
        assert np.allclose(got[:, 1] * f, want[:, 1], rtol=2e-3)
        assert np.abs(got[:, 2:] * f[:, None] - want[:, 2:]).max() <= 2e-3 * max(1.0, np.abs(want[:, 2:]).max())
        empty = parts[r][1].cpu().numpy()
        assert np.isneginf(empty[:, 0]).all() and not empty[:, 1:].any()
    allp = torch.stack(parts)                         # [2 shards][2 rows][64][130] == all-gather layout
    out = torch.zeros((2, 64, 128), dtype=torch.float32, device=cuda)
    ctxs[0].merge_partials(allp, 2, 2, 64, out)
    ctxs[0].sync()
    check_attention(out[0].cpu().numpy(), oracle.attention(q[0], Kf, Vf), "merged shards")
    assert not out[1].cpu().numpy().any()             # no keys anywhere -> zeros (hy3_gpu.cu:245)
    for c in ctxs:
        c.close()


def test_kv_head_shard_writes_only_its_heads(cuda, oracle):
    import torch
    from hy3_b200 import Hy3Attn
    n = 700
    K = oracle.fill_normal((n, 8, 128), SEED, 91)
    V = oracle.fill_normal((n, 8, 128), SEED, 92)
    q = oracle.fill_normal((1, 64, 128), SEED, 93)
    ctx = Hy3Attn(kv_dtype="int4", n_layers=1, kv_head_begin=2, kv_head_count=2, max_batch=1, max_tokens=1024)
    Kf, Vf = load_cache(ctx, oracle, "int4", 0, 0, K, V)
    ks, _ = ctx.export_kv(0, 0, 0, n)
    full = make_slots(oracle, K, "int4")
    assert np.array_equal(ks[:, 16 + 2 * 64:16 + 4 * 64], full[:, 16 + 2 * 64:16 + 4 * 64]) and not ks[:, 16:16 + 128].any()
    ctx.batch_set([0], [n - 1])
    out = torch.full((1, 64, 128), 7.0, dtype=torch.float32, device=cuda)
    ctx.decode(0, torch.from_numpy(q).to(cuda), out=out)
    ctx.sync()
    out = out.cpu().numpy()[0]
    want = oracle.attention(q[0], Kf, Vf)
    check_attention(out[16:32], want[16:32], "owned heads")
    assert (out[:16] == 7.0).all() and (out[32:] == 7.0).all()
    ctx.close()


@pytest.mark.parametrize("dt", ["int8", "int4"])
def test_one_kv_head_of_a_ragged_batch(cuda, oracle, dt):
    """A context that owns ONE KV head of 60 sequences (the KV-head shard of a ragged batch on 8 GPUs): fewer segments than
    CTAs, but so many that giving every segment whole CTAs would leave some CTAs with far more pages than others -- the
    kernel then takes the equal split over all units (CTAs straddle segments).  A fused step, checked per sequence."""
    import torch
    from hy3_b200 import Hy3Attn
    from hy3_b200.attn import decode_schedule
    rng = np.random.default_rng(11)
    lens0 = [int(x) for x in rng.integers(100, 6000, size=60)]
    B = len(lens0)
    # the host mirror of the schedule says: not the aligned split (ranges are equal to a page)
    sizes = [u1 - u0 for u0, u1 in (decode_schedule([n + 1 for n in lens0], 1, 148, c)[1:] for c in range(148))]
    assert max(sizes) - min(sizes) <= 1
    hb = 5
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, kv_head_begin=hb, kv_head_count=1, max_seqs=B, max_batch=B,
                  max_tokens=sum(lens0) + 256 * B, max_tokens_per_seq=8192)
    for s_, n0 in enumerate(lens0):
        ctx.fill_random(0, s_, 0, n0, 900 + s_)
    q = oracle.fill_normal((B, 64, 128), SEED, 431)
    k = oracle.fill_normal((B, 8, 128), SEED, 432)
    v = oracle.fill_normal((B, 8, 128), SEED, 433)
    tq, tk, tv = (torch.from_numpy(x).to(cuda) for x in (q, k, v))
    qo = torch.zeros((B, 64, 128), dtype=torch.float32, device=cuda)
    out = torch.full((B, 64, 128), 7.0, dtype=torch.float32, device=cuda)
    ctx.batch_set(list(range(B)), lens0)
    ctx.decode_step(0, tq, tk, tv, out=out, q_out=qo)
    ctx.sync()
    out, qo = out.cpu().numpy(), qo.cpu().numpy()
    assert (out[:, :8 * hb] == 7.0).all() and (out[:, 8 * hb + 8:] == 7.0).all()          # only the owned heads are written
    for s_ in range(0, B, 7):
        ks, vs = ctx.export_kv(0, s_, 0, lens0[s_] + 1)
        Kf, Vf = slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)
        want = oracle.attention(qo[s_], Kf, Vf)
        check_attention(out[s_][8 * hb:8 * hb + 8], want[8 * hb:8 * hb + 8], "seq %d len %d" % (s_, lens0[s_] + 1))
    ctx.close()


def test_errors_are_codes_not_exits(cuda, oracle):
    import torch
    from hy3_b200 import Hy3Attn, Hy3AttnError
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_batch=2, max_tokens=256)
    q = torch.zeros((1, 64, 128), dtype=torch.float32, device=cuda)
    assert ctx.lib.hy3a_decode(ctx.h, 0, q.data_ptr(), 8192, q.data_ptr(), 8192, None) == -5   # no batch set
    with pytest.raises(Hy3AttnError) as e:
        ctx.batch_set([0], [100000])                    # beyond the pool
    assert e.value.code == -2
    with pytest.raises(Hy3AttnError):
        ctx.batch_set([3], [0])                         # sequence out of range
    ctx.batch_set([0], [5])
    with pytest.raises(Hy3AttnError):
        ctx._chk(ctx.lib.hy3a_decode(ctx.h, 9, q.data_ptr(), 8192, q.data_ptr(), 8192, None))  # bad layer
    ctx.close()


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("lens,heads,sizes", [      # sizes: CTAs per segment with an FP16, INT8, INT4 cache
    ([129], (0, 8), (2, 2, 2)), ([300], (0, 8), (4, 2, 2)), ([640], (3, 5), (8, 2, 2)), ([900], (0, 8), (8, 2, 2)), ([2200], (0, 8), (8, 4, 8)),
    ([257, 1, 128], (0, 8), (4, 2, 2)), ([1500, 700], (6, 2), (8, 4, 4)), ([4200], (7, 1), (1, 8, 8)),
    ([200, 130, 256, 255, 129, 300, 384, 200, 140], (0, 8), (2, 2, 2)), ([900, 0, 700], (2, 1), (8, 2, 2)), ([1025] * 5, (4, 3), (8, 2, 4))])
def test_decode_clusters_equal_the_grid(cuda, oracle, dt, lens, heads, sizes, monkeypatch):
    """Steps of few segments run as clusters of 2, 4 or 8 CTAs per (row, KV head).  Fewer pages than CTAs, full and one-token last
    pages, rows without keys, several heads and rows: the sizes that the rule gives, against the oracle and the grid (a context
    without clusters), outputs and the cache; repeated launches bit for bit; partial records; the step captured into a graph and
    replayed for shorter and longer rows.  The two differ by the order of fp32 sums and fp16 digits of P (2^-22):
    2e-5 is over ten times that at outputs below 4."""
    import torch
    from hy3_b200 import Hy3Attn
    h0, nh = heads
    n = len(lens)
    rng = np.random.default_rng(5)
    q, k, v = (torch.from_numpy(rng.standard_normal((n, h, 128)).astype(np.float32)).to(cuda) for h in (64, 8, 8))
    res = []
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for clusters in (True, False):
        monkeypatch.setenv("HY3A_NO_CLUSTERS", str(int(not clusters)))
        ctx = Hy3Attn(kv_dtype=dt, n_layers=2, kv_head_begin=h0, kv_head_count=nh, max_seqs=n, max_batch=n, max_tokens=sum(lens) + 128 * n, max_tokens_per_seq=max(lens) + 128)
        for layer in range(2):
            for i, m in enumerate(lens):
                if m > 1:
                    ctx.fill_random(layer, i, 0, m - 1, 100 * layer + i)
        slots = [m - 1 for m in lens]
        ctx.batch_set(list(range(n)), slots)
        assert ctx.decode_cluster() == (sizes[("fp16", "int8", "int4").index(dt)] if clusters else 1) or sms != 148
        outs = []
        for _ in range(4):
            for layer in range(2):
                outs.append(ctx.decode_step(layer, q, k, v, out=torch.full((n, 64, 128), float("nan"), device=cuda)))
        part = torch.full((n, 8 * nh, 130), float("nan"), device=cuda)
        ctx.decode_step(0, q, k, v, partials=part)
        ctx.sync()
        assert all(torch.equal(outs[i][:, 8 * h0:8 * (h0 + nh)], outs[i % 2][:, 8 * h0:8 * (h0 + nh)]) for i in range(8))
        qn = torch.zeros((n, 64, 128), device=cuda)
        ctx.decode_step(0, q, k, v, q_out=qn)
        ctx.sync()
        kv = {i: ctx.export_kv(0, i, 0, m) for i, m in enumerate(lens) if m > 0}
        # a graph captured for these rows, replayed for shorter and for longer ones
        side = torch.cuda.Stream()
        g_out = torch.zeros((n, 64, 128), device=cuda)
        ctx.set_stream(side)
        with torch.cuda.stream(side):
            ctx.decode_step(1, q, k, v, out=g_out)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            ctx.decode_step(1, q, k, v, out=g_out)
        side.synchronize()
        ctx.use_torch_stream()
        replays = []
        for other in ([max(-1, m - 3) if m > 2 else m - 1 for m in lens], [m + 100 for m in lens]):
            ctx.batch_set(list(range(n)), other)
            graph.replay()
            ctx.sync()
            replays.append(g_out.clone())
        res.append((outs[0], outs[1], part, torch.stack(replays, 1), kv, qn))
        del graph
        ctx.close()
    own = slice(8 * h0, 8 * (h0 + nh))
    for a, b in zip(res[0][:2], res[1][:2]):
        assert torch.isfinite(a[:, own]).all() and (a[:, own] - b[:, own]).abs().max() < 2e-5
        assert torch.isnan(a[:, :8 * h0]).all() and torch.isnan(a[:, 8 * (h0 + nh):]).all()
    assert (res[0][3][:, :, own] - res[1][3][:, :, own]).abs().max() < 2e-5
    live = [i for i, m in enumerate(lens) if m > 0]
    for x in (0, 1):
        p = res[x][2][live]
        assert ((p[:, :, 2:] / p[:, :, 1:2]) - res[0][0][live][:, own]).abs().max() < 2e-5
        assert all((res[x][2][i, :, 1] == 0).all() and torch.isneginf(res[x][2][i, :, 0]).all() for i, m in enumerate(lens) if m == 0)
    for i in live:
        assert all(np.array_equal(a, b) for a, b in zip(res[0][4][i], res[1][4][i]))
        Kf, Vf = (slots_to_float(oracle, x, dt) for x in res[0][4][i])
        want = oracle.attention(res[0][5][i].cpu().numpy(), Kf, Vf)
        check_attention(res[0][0][i, own].cpu().numpy(), want[own], "%s row %d of %d tokens" % (dt, i, lens[i]))


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("n,heads", [(3201, (7, 1)), (20000, (3, 1)), (33000, (2, 2))])
def test_decode_few_heads_long_row(cuda, oracle, dt, n, heads):
    """Few KV heads with long rows: segments of as many pieces as their bound allows, on fewer CTAs than the GPU has."""
    import torch
    from hy3_b200 import Hy3Attn
    h0, nh = heads
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, kv_head_begin=h0, kv_head_count=nh, max_batch=1, max_tokens=n + 128)
    ctx.fill_random(0, 0, 0, n, 31)
    q = oracle.fill_normal((64, 128), SEED, 811)
    ctx.batch_set([0], [n - 1])
    outs = [ctx.decode(0, torch.from_numpy(q[None]).to(cuda)) for _ in range(5)]
    ctx.sync()
    ks, vs = ctx.export_kv(0, 0, 0, n)
    ctx.close()
    own = slice(8 * h0, 8 * (h0 + nh))
    assert all(torch.equal(o, outs[0]) for o in outs)
    want = oracle.attention_f64(q, slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)).astype(np.float32)
    check_attention(outs[0][0, own].cpu().numpy(), want[own], "%s %d tokens, %d heads" % (dt, n, nh))


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("lens,heads", [([0], (0, 8)), ([0, 0, 0], (5, 3)), ([1, 0, 0], (0, 1)), ([20000] + [0] * 29, (3, 1))])
def test_rows_without_keys_are_written(cuda, dt, lens, heads):
    """A row with slot -1 gets zero outputs, or empty records {-inf, 0, 0...}, also where the CTA it belongs to has no pages, where no CTA
    has any, and in a captured step whose rows lose their keys before the replay.  Buffers start as NaN; heads of others stay."""
    import torch
    from hy3_b200 import Hy3Attn
    h0, nh = heads
    n = len(lens)
    own = slice(8 * h0, 8 * (h0 + nh))
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, kv_head_begin=h0, kv_head_count=nh, max_seqs=n, max_batch=n, max_tokens=sum(lens) + 128 * n, max_tokens_per_seq=max(lens) + 128)
    for i, m in enumerate(lens):
        if m:
            ctx.fill_random(0, i, 0, m, 7 + i)
    q = torch.randn((n, 64, 128), device=cuda, generator=torch.Generator(cuda).manual_seed(1))

    def fresh():
        return torch.full((n, 64, 128), float("nan"), device=cuda), torch.full((n, 8 * nh, 130), float("nan"), device=cuda)

    def check(out, part, empty):
        assert not torch.isnan(out[:, own]).any() and not torch.isnan(part).any()
        assert torch.isnan(out[:, :8 * h0]).all() and torch.isnan(out[:, 8 * (h0 + nh):]).all()
        for i in range(n):
            assert (i in empty) == (not out[i, own].any().item())
            assert (i in empty) == (torch.isneginf(part[i, :, 0]).all().item() and not part[i, :, 1:].any().item())

    ctx.batch_set(list(range(n)), [m - 1 for m in lens])
    out, part = fresh()
    ctx.decode(0, q, out=out)
    ctx.decode(0, q, partials=part)
    ctx.sync()
    check(out, part, [i for i, m in enumerate(lens) if m == 0])
    # captured with one key more in every row, replayed with these rows and with none that has keys
    ctx.batch_set(list(range(n)), lens)
    ctx.sync()
    side, (g_out, g_part) = torch.cuda.Stream(), fresh()
    ctx.set_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ctx.decode(0, q, out=g_out)
        ctx.decode(0, q, partials=g_part)
    side.synchronize()
    ctx.use_torch_stream()
    for slots in ([m - 1 for m in lens], [-1] * n):
        ctx.batch_set(list(range(n)), slots)
        g_out.fill_(float("nan"))
        g_part.fill_(float("nan"))
        graph.replay()
        ctx.sync()
        check(g_out, g_part, [i for i, s in enumerate(slots) if s < 0])
    del graph
    ctx.close()


def test_largest_batch_keeps_the_page_ring(cuda):
    """The largest FP16 batch whose page counts fit beside a ring of two pages: the fused step needs no q_out there (it does without a
    ring), and rows at both ends equal those of a small context (the two differ by the order of fp32 sums: 2e-5, as between cluster
    and grid)."""
    import torch
    from hy3_b200 import Hy3Attn
    n = 12543
    rows = [0, 1, 6000, n - 2, n - 1]
    slots = np.arange(n) % 260
    q = torch.randn((n, 64, 128), device=cuda, generator=torch.Generator(cuda).manual_seed(2))
    res = []
    for idx in (np.arange(n), np.array(rows)):
        ctx = Hy3Attn(kv_dtype="fp16", n_layers=1, max_batch=len(idx), max_tokens=384)
        ctx.fill_random(0, 0, 0, 384, 5)
        ctx.batch_set([0] * len(idx), slots[idx], idx)
        res.append(ctx.decode_step(0, q[torch.from_numpy(idx).to(cuda)], None, None))
        ctx.sync()
        ctx.close()
    assert torch.isfinite(res[0]).all() and (res[0][rows] - res[1]).abs().max() < 2e-5


@pytest.mark.parametrize("dt,kind", [("fp16", "nan"), ("fp16", "+inf"), ("int8", "nan"), ("int4", "nan")])
def test_decode_non_finite_scores(cuda, dt, kind):
    """A key whose score is NaN or +inf makes the outputs of its KV head's queries NaN, whichever piece it is in, and no others: in one
    piece, as a cluster, in pieces whose records are folded, captured, through partial records, and with two rows."""
    import torch
    from hy3_b200 import Hy3Attn
    for ntok, at in ((1, 0), (100, 3), (641, 640), (700, 650), (3000, 0), (5000, 2222), (40000, 39999), (40000, 20000)):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=2, max_batch=2, max_tokens=2 * ntok + 128, max_tokens_per_seq=40960)
        for i in range(2):
            ctx.fill_random(0, i, 0, ntok, 5 + i)
        ks, vs = ctx.export_kv(0, 0, at, 1)
        ks[0].view(np.float16)[3 * 128 if dt == "fp16" else 3] = np.float16(kind)       # KV head 3: an element of the key, or its scale
        ctx.import_kv(0, 0, at, ks, vs)
        q = torch.randn((2, 64, 128), device=cuda, generator=torch.Generator(cuda).manual_seed(1))
        q[:, :, 0] = 1.0                                                                # the score of the infinite element is +inf
        outs = []
        for rows in ([0], [0, 1]):
            n = len(rows)
            ctx.batch_set(rows, [ntok - 1] * n)
            outs.append(ctx.decode(0, q[:n]))
            part = torch.zeros((n, 64, 130), device=cuda)
            ctx.decode(0, q[:n], partials=part)
            merged = torch.zeros((n, 64, 128), device=cuda)
            ctx.merge_partials(part, 1, n, 64, merged)
            outs.append(merged)
            ctx.sync()
            side, graph, g_out = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros((n, 64, 128), device=cuda)
            torch.cuda.synchronize()
            ctx.set_stream(side)
            with torch.cuda.graph(graph, stream=side):
                ctx.decode(0, q[:n], out=g_out)
            ctx.use_torch_stream()
            graph.replay()
            ctx.sync()
            outs.append(g_out)
            del graph
        ctx.close()
        for o in outs:
            assert torch.isnan(o[0, 24:32]).all(), "%d tokens, key %d: dropped" % (ntok, at)
            assert torch.isfinite(o[0, :24]).all() and torch.isfinite(o[0, 32:]).all() and torch.isfinite(o[1:]).all()


@pytest.mark.parametrize("dt", ["int8", "int4"])
@pytest.mark.parametrize("heads", [1, 8])
@pytest.mark.parametrize("no_clusters", ["1", "0"])
def test_pieces_whose_scores_are_all_minus_infinity(cuda, oracle, dt, heads, no_clusters, monkeypatch):
    """Keys whose scores are -inf weigh nothing, and a piece that holds no others (denominator 0) is skipped on every route: infinite V
    scales beside such keys, which make 0 x infinity of the piece's sums, do not reach the output."""
    import torch
    from hy3_b200 import Hy3Attn
    monkeypatch.setenv("HY3A_NO_CLUSTERS", no_clusters)
    n, cut = 2048, 1024                                 # pieces of one page in the grid, of four in a cluster: both end at the cut
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, kv_head_count=heads, max_tokens=n + 128)
    ctx.fill_random(0, 0, 0, n, 3)
    ks, vs = ctx.export_kv(0, 0, 0, n)
    want_k, want_v = slots_to_float(oracle, ks[cut:].copy(), dt), slots_to_float(oracle, vs[cut:].copy(), dt)
    ks[:cut, :16].view(np.float16)[:] = -np.inf
    vs[:cut, :16].view(np.float16)[:] = np.inf
    ks[:cut, 16:] = 1 if dt == "int8" else 0x11         # positive codes and queries: every score is -inf
    ctx.import_kv(0, 0, 0, ks, vs)
    q = np.abs(oracle.fill_normal((1, 64, 128), SEED, 451)) + 0.1
    ctx.batch_set([0], [n - 1])
    assert (ctx.decode_cluster() > 1) == (no_clusters == "0")
    out = ctx.decode(0, torch.from_numpy(q.astype(np.float32)).to(cuda))
    ctx.sync()
    want = oracle.attention(q[0].astype(np.float32), want_k, want_v)
    check_attention(out[0, :8 * heads].cpu().numpy(), want[:8 * heads], "%s, %d heads" % (dt, heads))
    ctx.close()


@pytest.mark.parametrize("lens,heads,sizes", [      # CTAs per segment with an FP16, INT8, INT4 cache
    ([128], 8, (1, 1, 1)), ([129] * 9, 8, (2, 2, 2)), ([129] * 10, 8, (1, 1, 1)), ([9216], 8, (1, 8, 8)), ([9217], 8, (1, 1, 8)), ([12000], 8, (1, 1, 8)),
    ([14000], 8, (1, 1, 1)), ([5000] * 2, 8, (1, 4, 4)), ([5000] * 3, 8, (1, 1, 4)), ([8000] * 3, 8, (1, 1, 1)), ([8000] * 4, 8, (4, 1, 4)),
    ([6000] * 30, 1, (4, 4, 4)), ([20000], 8, (1, 1, 1))])
def test_decode_cluster_rule(cuda, lens, heads, sizes):
    """Where the rule takes clusters and where the grid, on 148 SMs (74 / 33 / 15 clusters of 2 / 4 / 8 at once)."""
    import torch
    from hy3_b200 import Hy3Attn
    for dt, size in zip(("fp16", "int8", "int4"), sizes):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, kv_head_count=heads, max_seqs=len(lens), max_batch=len(lens), max_tokens=sum(lens) + 128 * len(lens), max_tokens_per_seq=max(lens))
        ctx.batch_set(list(range(len(lens))), [m - 1 for m in lens])
        assert ctx.decode_cluster() == size or torch.cuda.get_device_properties(0).multi_processor_count != 148, dt
        ctx.sync()
        ctx.close()
