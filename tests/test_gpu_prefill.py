"""GPU parity of the tcgen05 chunk-prefill attention (through the C ABI) against the oracle's causal
prefill -- one decode attention per query over the keys [0, base+i] (restatement of hy3_gpu.cu:379-412 /
hy3.c:617-652) -- evaluated on the SAME stored K/V and the same fp16 queries."""
import numpy as np
import pytest

from helpers import SEED, check_attention, make_slots, slots_to_float

pytestmark = pytest.mark.gpu


def run_case(cuda, oracle, dt, base, nq, rows=None, eps=1e-6, cluster=None):
    import torch
    from hy3_b200 import Hy3Attn
    ntok = base + nq
    ctx = Hy3Attn(kv_dtype=dt, n_layers=2, max_batch=max(nq, base, 1), max_tokens=ntok + 256, rms_eps=eps)
    assert cluster is None or ctx.prefill_cluster(base, nq) == cluster
    w = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    ctx.set_norm_weights(1, w[0], w[1])
    q = oracle.fill_normal((ntok, 64, 128), SEED, 501)
    k = oracle.fill_normal((ntok, 8, 128), SEED, 502)
    v = oracle.fill_normal((ntok, 8, 128), SEED, 503)
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    if base:                                                  # an earlier turn / earlier chunks
        ctx.batch_set([0] * base, list(range(base)))
        ctx.append(1, tq[:base], tk[:base], tv[:base])
    ctx.batch_set([0] * nq, list(range(base, ntok)))
    q16 = torch.empty((nq, 64, 128), dtype=torch.float16, device=cuda)
    ctx.append(1, tq[base:], tk[base:], tv[base:], q_out16=q16)
    out = ctx.prefill(1, 0, base, q16)
    ctx.sync()
    ks, vs = ctx.export_kv(1, 0, 0, ntok)
    Kf, Vf = slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)
    qf = q16.float().cpu().numpy()
    out = out.cpu().numpy()
    rows = list(range(nq)) if rows is None else rows
    want = oracle.prefill_causal(qf, Kf, Vf, base, rows=rows)
    worst = 0.0
    for i in rows:
        err, _ = check_attention(out[i], want[i], "%s base=%d nq=%d row %d" % (dt, base, nq, i))
        worst = max(worst, err)
    ctx.close()
    return worst


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("base,nq", [(0, 1), (0, 16), (0, 40), (0, 129), (100, 28), (127, 130), (256, 256)])
def test_prefill_small(cuda, oracle, dt, base, nq):
    worst = run_case(cuda, oracle, dt, base, nq)
    print("prefill %s base=%d nq=%d worst max-abs %.3g" % (dt, base, nq, worst))


@pytest.mark.parametrize("dt", ["fp16", "int8"])
def test_prefill_chunk_over_prefix(cuda, oracle, dt):
    """A 512-token chunk on top of a 1536-token prefix; sampled rows at the chunk and tile boundaries."""
    run_case(cuda, oracle, dt, 1536, 512, rows=[0, 1, 15, 16, 127, 128, 255, 256, 500, 511])


@pytest.mark.parametrize("dt", ["fp16", "int8", "int4"])
@pytest.mark.parametrize("base,nq", [(2047, 1), (3970, 45), (4090, 37), (4060, 129), (3999, 33)])
def test_prefill_cut_along_the_keys(cuda, oracle, dt, base, nq, monkeypatch):
    """Chunks whose blocks are cut into several pieces (records + fold; not as clusters): warps without queries, rows whose keys in the
    last piece are all masked, odd bases."""
    from hy3_b200.attn import prefill_schedule
    monkeypatch.setenv("HY3A_NO_CLUSTERS", "1")
    assert (prefill_schedule(base, nq, 8)[:, 5] > 1).any()
    run_case(cuda, oracle, dt, base, nq, cluster=1, rows=sorted({0, nq // 2, max(nq - 2, 0), nq - 1, min(31, nq - 1), min(32, nq - 1)}))


@pytest.mark.parametrize("kind", ["nan", "+inf", "-inf"])
@pytest.mark.parametrize("base,nq,first,clusters", [(0, 96, 16, False), (4060, 37, 4000, False), (4060, 37, 4000, True), (1001, 40, 970, True)])
def test_prefill_non_finite_scores(cuda, oracle, base, nq, first, clusters, kind, monkeypatch):
    """A key whose score is NaN or +inf makes every query that sees it NaN, wherever the key lies in a step (64 positions), uncut,
    cut and in a cluster; a score of -inf is a weight of 0.  Against softmax in 64 bits."""
    if not clusters:
        monkeypatch.setenv("HY3A_NO_CLUSTERS", "1")
    import torch
    from hy3_b200 import Hy3Attn
    from hy3_b200.attn import prefill_schedule
    assert clusters or (len(prefill_schedule(base, nq, 8)) > 0) == (base > 0)
    ntok = base + nq
    q = oracle.fill_normal((nq, 64, 128), SEED, 521).astype(np.float16)
    q[:, :, 0] = 1.0
    k = oracle.fill_normal((ntok, 8, 128), SEED, 522).astype(np.float16)
    v = oracle.fill_normal((ntok, 8, 128), SEED, 523)
    vs = make_slots(oracle, v, "fp16")
    tq = torch.from_numpy(q).to(cuda)
    ctx = Hy3Attn(kv_dtype="fp16", n_layers=1, max_batch=max(nq, 16), max_tokens=ntok + 128)
    assert (ctx.prefill_cluster(base, nq) > 1) == clusters
    v64 = v.astype(np.float16).astype(np.float64)
    seen = np.arange(ntok)[None, :] <= base + np.arange(nq)[:, None]
    for r in range(8):
        kk = k.copy()
        for h in range(8):                                    # a key of its own for every KV head
            kk[first + 8 * r + h, h, 0] = np.float16(kind)
        ctx.import_kv(0, 0, 0, np.ascontiguousarray(kk).view(np.uint8).reshape(ntok, 2048), vs)
        out = ctx.prefill(0, 0, base, tq)
        ctx.sync()
        out = out.cpu().numpy()
        for h in range(8):
            s = np.einsum("qgd,td->qgt", q[:, 8 * h:8 * h + 8].astype(np.float64), kk[:, h].astype(np.float64)) / np.sqrt(128.0)
            s = np.where(seen[:, None, :], s, -np.inf)
            with np.errstate(invalid="ignore"):
                w = np.exp(s - s.max(axis=2, keepdims=True))
            want = np.einsum("qgt,td->qgd", w / w.sum(axis=2, keepdims=True), v64[:, h])
            got = out[:, 8 * h:8 * h + 8]
            hit = base + np.arange(nq) >= first + 8 * r + h
            what = "%s at key %d" % (kind, first + 8 * r + h)
            if kind != "-inf":
                assert np.isnan(want[hit]).all() and np.isnan(got[hit]).all(), what + ": the key was dropped"
                got, want = got[~hit], want[~hit]
            if len(got):
                check_attention(got, want, what)
    ctx.close()


@pytest.mark.parametrize("dt,base,nq,heads,cut", [
    ("fp16", 0, 2048, (0, 8), False), ("int8", 2048, 953, (0, 8), False), ("int4", 40, 700, (0, 8), False), ("fp16", 9930, 97, (0, 8), True),
    ("int8", 1001, 512, (2, 4), True), ("fp16", 500, 1000, (6, 2), True), ("int4", 3000, 200, (7, 1), True), ("fp16", 3000, 300, (5, 3), True),
    ("int8", 100, 2900, (4, 3), False)])
def test_prefill_every_block_and_head(cuda, oracle, dt, base, nq, heads, cut, monkeypatch):
    """Grids (no clusters) in several groups of blocks (more CTAs than SMs) with a ragged last group, uncut and cut, and contexts that own some of
    the KV heads: one query of every 32-token block, every owned head, into an output that starts as NaN; heads of others are not
    written.  Repeated and interleaved with a chunk of another shape on the same records: identical bits."""
    import torch
    from hy3_b200 import Hy3Attn
    from hy3_b200.attn import prefill_schedule
    monkeypatch.setenv("HY3A_NO_CLUSTERS", "1")
    h0, nh = heads
    plan = prefill_schedule(base, nq, nh)
    assert (len(plan) > 0) == cut
    ntok = base + nq
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=nq, max_tokens=ntok + 128, kv_head_begin=h0, kv_head_count=nh)
    ctx.fill_random(0, 0, 0, ntok, 77)
    q16 = torch.from_numpy(oracle.fill_normal((nq, 64, 128), SEED, 531).astype(np.float16)).to(cuda)
    outs = []
    for _ in range(3):
        outs.append(ctx.prefill(0, 0, base, q16, out=torch.full((nq, 64, 128), float("nan"), device=cuda)))
        ctx.prefill(0, 0, ntok - 33, q16[:33])
    ctx.sync()
    ks, vs = ctx.export_kv(0, 0, 0, ntok)
    ctx.close()
    own = slice(8 * h0, 8 * (h0 + nh))
    assert all(torch.equal(o[:, own], outs[0][:, own]) for o in outs[1:])
    assert torch.isfinite(outs[0][:, own]).all()
    assert torch.isnan(outs[0][:, :8 * h0]).all() and torch.isnan(outs[0][:, 8 * (h0 + nh):]).all()
    rows = sorted({min(32 * b + (7 * b) % 32, nq - 1) for b in range(-(-nq // 32))} | {0, nq - 1})
    Kf, Vf = slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)
    want = oracle.prefill_causal(q16.float().cpu().numpy(), Kf, Vf, base, rows=rows)
    got = outs[0].cpu().numpy()
    for i in rows:
        for h in range(h0, h0 + nh):
            check_attention(got[i, 8 * h:8 * h + 8], want[i, 8 * h:8 * h + 8], "%s base=%d nq=%d row %d KV head %d" % (dt, base, nq, i, h))


@pytest.mark.parametrize("dt,base,nq,heads,size", [
    ("fp16", 1001, 1, (0, 8), 8), ("int8", 0, 500, (0, 2), 2), ("int4", 449, 31, (0, 8), 2), ("fp16", 1001, 45, (0, 8), 4),
    ("int8", 1000, 200, (0, 8), 2), ("int4", 4064, 32, (0, 8), 8), ("fp16", 900, 33, (3, 5), 4), ("int8", 2500, 70, (7, 1), 8),
    ("fp16", 0, 1200, (6, 1), 2), ("int4", 40, 900, (2, 1), 4)])
def test_prefill_clusters(cuda, oracle, dt, base, nq, heads, size):
    """Blocks shared by the CTAs of a cluster: tokens that fill no softmax warp, one, or the last partly; fewer steps than CTAs (pieces
    without keys, or with masked ones only); several heads and blocks per launch; every owned row finite and the others untouched;
    one query per 4 tokens against the oracle; repeated launches bit for bit; a context without records takes the same path."""
    import torch
    from hy3_b200 import Hy3Attn
    h0, nh = heads
    ntok = base + nq
    q16 = torch.from_numpy(oracle.fill_normal((nq, 64, 128), SEED, 551).astype(np.float16)).to(cuda)
    outs = []
    for batch in (max(nq, 16), 8):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=batch, max_tokens=ntok + 128, kv_head_begin=h0, kv_head_count=nh)
        ctx.fill_random(0, 0, 0, ntok, 79)
        assert ctx.prefill_cluster(base, nq) == size or torch.cuda.get_device_properties(0).multi_processor_count != 148
        for _ in range(3):
            outs.append(ctx.prefill(0, 0, base, q16, out=torch.full((nq, 64, 128), float("nan"), device=cuda)))
        ctx.sync()
        ks, vs = ctx.export_kv(0, 0, 0, ntok)
        ctx.close()
    own = slice(8 * h0, 8 * (h0 + nh))
    assert all(torch.equal(o[:, own], outs[0][:, own]) for o in outs[1:3]) and all(torch.equal(o[:, own], outs[3][:, own]) for o in outs[4:])
    assert all(torch.isfinite(o[:, own]).all() for o in outs)
    assert torch.isnan(outs[0][:, :8 * h0]).all() and torch.isnan(outs[0][:, 8 * (h0 + nh):]).all()
    rows = sorted({min(4 * b + b % 4, nq - 1) for b in range(-(-nq // 4))} | {0, nq - 1})
    want = oracle.prefill_causal(q16.float().cpu().numpy(), slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt), base, rows=rows)
    for o in (outs[0], outs[3]):
        got = o.cpu().numpy()
        for i in rows:
            check_attention(got[i, own], want[i, own], "%s base=%d nq=%d row %d" % (dt, base, nq, i))


@pytest.mark.parametrize("dt,base,nq,heads", [("fp16", 0, 33, (0, 8)), ("int8", 30, 48, (0, 8)), ("int4", 0, 288, (0, 8)), ("int8", 0, 289, (0, 8)), ("fp16", 0, 49, (2, 3))])
def test_prefill_uncut_blocks_of_one_tile(cuda, oracle, dt, base, nq, heads, monkeypatch):
    """Uncut grids whose blocks of 16 tokens fit at once (up to 288 tokens of 8 heads), with a last block of one token and a full one; one token more."""
    test_prefill_every_block_and_head(cuda, oracle, dt, base, nq, heads, False, monkeypatch)


@pytest.mark.parametrize("dt,base,nq,heads", [("fp16", 700, 15, (0, 8)), ("int8", 1001, 16, (0, 8)), ("int4", 1001, 17, (0, 8)), ("fp16", 3000, 64, (0, 8)), ("int8", 2000, 65, (2, 3))])
def test_prefill_clusters_of_one_tile(cuda, oracle, dt, base, nq, heads):
    """Blocks of 16 tokens: a last block of one token, of 15 and a full one, several blocks per head."""
    from hy3_b200 import Hy3Attn
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=nq, max_tokens=base + nq, kv_head_begin=heads[0], kv_head_count=heads[1])
    size = ctx.prefill_cluster(base, nq)
    ctx.close()
    assert size > 1
    test_prefill_clusters(cuda, oracle, dt, base, nq, heads, size)


@pytest.mark.parametrize("base,nq,heads,size", [
    (100, 8, 8, 1), (500, 2, 4, 8), (8192, 2, 8, 8), (8192, 45, 8, 4), (16000, 2, 8, 1), (16000, 8, 8, 1), (16000, 30, 8, 8), (16000, 200, 8, 1), (16000, 256, 8, 2),
    (30000, 8, 8, 1), (30000, 30, 8, 1), (4064, 300, 4, 1), (16000, 2048, 8, 2)])
def test_prefill_cluster_rule(cuda, base, nq, heads, size):
    """Where the rule takes clusters and where records or whole blocks, on 148 SMs (74 / 33 / 15 clusters of 2 / 4 / 8 at once)."""
    import torch
    from hy3_b200 import Hy3Attn
    ctx = Hy3Attn(kv_dtype="int4", n_layers=1, max_batch=max(16, nq), max_tokens=base + nq, kv_head_count=heads)
    assert ctx.prefill_cluster(base, nq) == size or torch.cuda.get_device_properties(0).multi_processor_count != 148
    ctx.close()


@pytest.mark.parametrize("dt,base,nq,heads", [("int8", 2500, 500, (3, 5)), ("int4", 500, 1500, (2, 2)), ("fp16", 4500, 150, (0, 8))])
def test_prefill_records_where_no_cluster_pays(cuda, oracle, dt, base, nq, heads, monkeypatch):
    """Chunks that still leave records: the checks of the grids above."""
    from hy3_b200 import Hy3Attn
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=nq, max_tokens=base + nq, kv_head_begin=heads[0], kv_head_count=heads[1])
    assert ctx.prefill_cluster(base, nq) == 1
    ctx.close()
    test_prefill_every_block_and_head(cuda, oracle, dt, base, nq, heads, True, monkeypatch)


def test_prefill_without_records(cuda, oracle, monkeypatch):
    """A context without piece records (max_batch < 16) runs uncut what another one cuts (where neither takes clusters)."""
    import torch
    from hy3_b200 import Hy3Attn
    from hy3_b200.attn import prefill_schedule
    monkeypatch.setenv("HY3A_NO_CLUSTERS", "1")
    base, nq = 3970, 45
    assert len(prefill_schedule(base, nq, 8)) > 0 and len(prefill_schedule(base, nq, 8, 148, 0)) == 0
    q16 = torch.from_numpy(oracle.fill_normal((nq, 64, 128), SEED, 541).astype(np.float16)).to(cuda)
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_batch=8, max_tokens=4096 + 128)
    ctx.fill_random(0, 0, 0, base + nq, 78)
    out = ctx.prefill(0, 0, base, q16)
    ctx.sync()
    ks, vs = ctx.export_kv(0, 0, 0, base + nq)
    ctx.close()
    rows = [0, 15, 16, 31, 32, 44]
    want = oracle.prefill_causal(q16.float().cpu().numpy(), slots_to_float(oracle, ks, "int8"), slots_to_float(oracle, vs, "int8"), base, rows=rows)
    for i in rows:
        check_attention(out[i].cpu().numpy(), want[i], "row %d" % i)


def _chunked(cuda, oracle, dt, chunks, mirror_mb, monkeypatch, redo=None):
    """Feeds `chunks` (token counts) one after the other through append + prefill on ONE context; `redo` =
    (keep_ntok, n): after the last chunk the sequence is cut back to keep_ntok tokens and n DIFFERENT tokens follow.
    Returns the outputs of all prefill calls and the exported cache."""
    import torch
    from hy3_b200 import Hy3Attn
    if mirror_mb is None:
        monkeypatch.delenv("HY3A_PF_MIRROR_MB", raising=False)
    else:
        monkeypatch.setenv("HY3A_PF_MIRROR_MB", str(mirror_mb))
    total = sum(chunks)
    ctx = Hy3Attn(kv_dtype=dt, n_layers=2, max_batch=max(max(chunks), (redo or (0, 1))[1]), max_tokens=total + 512)
    q = oracle.fill_normal((total + 512, 64, 128), SEED, 511)
    k = oracle.fill_normal((total + 512, 8, 128), SEED, 512)
    v = oracle.fill_normal((total + 512, 8, 128), SEED, 513)
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    outs, base = [], 0
    steps = [(c, 0) for c in chunks]
    for n, shift in steps + ([(redo[1], 256)] if redo else []):
        if shift:                                            # cut back, then other tokens at the same slots
            base = redo[0]
            ctx.seq_release(0, base)
        ctx.batch_set([0] * n, list(range(base, base + n)))
        q16 = torch.empty((n, 64, 128), dtype=torch.float16, device=cuda)
        src = slice(base + shift, base + shift + n)
        ctx.append(1, tq[src], tk[src], tv[src], q_out=False, q_out16=q16)
        out = ctx.prefill(1, 0, base, q16)
        ctx.sync()
        outs.append((base, n, q16.float().cpu().numpy(), out.cpu().numpy()))
        base += n
    ks, vs = ctx.export_kv(1, 0, 0, base)
    ctx.close()
    return outs, ks, vs


@pytest.mark.parametrize("dt", ["fp16", "int8"])
def test_prefill_chunks_reuse_converted_pages(cuda, oracle, dt, monkeypatch):
    """Successive chunks convert only the pages they appended (the per-layer fp16 operand mirror).  The outputs must
    equal, bit for bit, those of a context that rebuilds the operands on every call, and must match the oracle also
    after the sequence was cut back and continued with different tokens (a stale mirror would show there)."""
    chunks, redo = [100, 156, 300, 84, 200], (300, 170)
    a, ks, vs = _chunked(cuda, oracle, dt, chunks, None, monkeypatch, redo)
    b, ks0, vs0 = _chunked(cuda, oracle, dt, chunks, 0, monkeypatch, redo)
    assert np.array_equal(ks, ks0) and np.array_equal(vs, vs0)
    for (base, n, _, oa), (_, _, _, ob) in zip(a, b):
        assert np.array_equal(oa, ob), "chunk at %d differs between mirrored and rebuilt operands" % base
    # oracle: the last call (after the cut) sees exactly the exported cache
    base, n, qf, out = a[-1]
    Kf, Vf = slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt)
    rows = [0, 1, 27, 28, 100, n - 1]
    want = oracle.prefill_causal(qf, Kf, Vf, base, rows=rows)
    for i in rows:
        check_attention(out[i], want[i], "%s after cut: base=%d row %d" % (dt, base, i))
    # and one call before the cut, against the cache as it was then = the same slots below its end (those below the
    # cut were not rewritten; only check a chunk that ends at or below the cut)
    base, n, qf, out = a[1]
    assert base + n <= redo[0]
    want = oracle.prefill_causal(qf, Kf, Vf, base, rows=[0, n - 1])
    for i in (0, n - 1):
        check_attention(out[i], want[i], "%s before cut: base=%d row %d" % (dt, base, i))


@pytest.mark.parametrize("dt", ["fp16", "int8"])
def test_append_twice_refreshes_operands(cuda, oracle, dt):
    """The same batch appended a second time with other K/V (no new hy3a_batch_set in between): the chunk attention
    must see the second version, i.e. the kept fp16 operands of the layer may not go stale."""
    import torch
    from hy3_b200 import Hy3Attn
    n = 200
    ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=n, max_tokens=512)
    q = oracle.fill_normal((n, 64, 128), SEED, 901)
    kv = [(oracle.fill_normal((n, 8, 128), SEED, 902 + 2 * i), oracle.fill_normal((n, 8, 128), SEED, 903 + 2 * i)) for i in range(2)]
    tq = torch.from_numpy(q).to(cuda)
    q16 = torch.empty((n, 64, 128), dtype=torch.float16, device=cuda)
    ctx.batch_set([0] * n, list(range(n)))
    for k, v in kv:
        ctx.append(0, tq, torch.from_numpy(k).to(cuda), torch.from_numpy(v).to(cuda), q_out=False, q_out16=q16)
        out = ctx.prefill(0, 0, 0, q16)
    ctx.sync()
    ks, vs = ctx.export_kv(0, 0, 0, n)
    rows = [0, 1, 100, n - 1]
    want = oracle.prefill_causal(q16.float().cpu().numpy(), slots_to_float(oracle, ks, dt), slots_to_float(oracle, vs, dt), 0, rows=rows)
    out = out.cpu().numpy()
    for i in rows:
        check_attention(out[i], want[i], "%s second append, row %d" % (dt, i))
    ctx.close()
