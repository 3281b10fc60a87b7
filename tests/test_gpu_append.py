"""GPU parity of the fused QK-RMSNorm + RoPE + KV quantise/append kernel, through the C ABI.

 - q/k after norm+RoPE vs the oracle (CPU restatement of hy3.c:435-444, :585-615): <= 1e-5 relative
   to max(1, |x|) (rsqrtf and device cosf/sinf differ from glibc by ulps).
 - codes and scales BIT-EXACT vs the oracle quantiser on identical fp32 inputs (V directly; K by
   routing the K rows through the Q path as well, which returns the device's own fp32 values).
 - codes and scales BIT-EXACT vs the reference's own CUDA quantiser kernels when oracle/_ref is
   present, and vs the committed fixture tests/golden/ref_gpu.npz when that exists.
"""
import os

import numpy as np
import pytest

from helpers import SEED, make_slots

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

POS = [0, 1, 2, 63, 64, 127, 128, 129, 4095, 4096, 32767, 262143, 262144, 1048575, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14]


def torch_rows(cuda, n, heads, seed=1):
    import torch
    return torch.randn((n, heads, 128), device=cuda, generator=torch.Generator(cuda).manual_seed(seed + heads))


def run_append(cuda, oracle, dt, eps, q, k, v, qw, kw, pos, table=None, probes=(1, 0, 0)):
    import torch
    from hy3_b200 import Hy3Attn
    n = q.shape[0]
    ctx = Hy3Attn(kv_dtype=dt, n_layers=2, max_batch=n, max_tokens=max(256, n + 128), rms_eps=eps)
    inv, af = table if table is not None else oracle.rope_table()
    ctx.set_rope(inv, af, *probes)
    ctx.set_norm_weights(1, qw, kw)
    ctx.batch_set([0] * n, list(range(n)), pos)
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    q16 = torch.empty((n, 64, 128), dtype=torch.float16, device=cuda)
    qo = ctx.append(1, tq, tk, tv, q_out16=q16)
    ctx.sync()
    ks, vs = ctx.export_kv(1, 0, 0, n)
    ks0, vs0 = ctx.export_kv(0, 0, 0, n)      # the other layer must be untouched
    assert not ks0.any() and not vs0.any()
    out = qo.cpu().numpy(), q16.cpu().numpy(), ks, vs
    ctx.close()
    return out


@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
@pytest.mark.parametrize("eps", [1e-5, 1e-6])
def test_append_matches_oracle(cuda, oracle, dt, eps):
    n = len(POS)
    q = oracle.fill_normal((n, 64, 128), SEED, 31)
    k = oracle.fill_normal((n, 8, 128), SEED, 32)
    v = oracle.fill_normal((n, 8, 128), SEED, 33)
    v[0] = 0.0                               # absmax 0 -> scale 1e-8 -> fp16 0, codes 0 (hy3_gpu.cu:260)
    v[1, 0] = np.arange(128, dtype=np.float32) - 63.5   # exact .5 ties
    v[2] *= 1e4
    w = (1.0 + 0.02 * oracle.fill_normal((128,), SEED, 34)).astype(np.float32)
    q[:, :8] = k                              # K rows also go through the Q path (same weights) -> device fp32 K
    inv, af = oracle.rope_table()
    qo, q16, ks, vs = run_append(cuda, oracle, dt, eps, q, k, v, w, w, POS)
    for i, p in enumerate(POS):
        oq, ok = oracle.qk_norm_rope(q[i], k[i], w, w, eps, p, inv, af)
        tol = 1e-5 * np.maximum(1.0, np.abs(oq))
        assert (np.abs(qo[i] - oq) <= tol).all(), "row %d pos %d: %.3g" % (i, p, np.abs(qo[i] - oq).max())
    assert np.array_equal(q16, qo.astype(np.float16))
    # V: raw fp32 -> quantiser, bit-exact against the oracle
    assert np.array_equal(vs, make_slots(oracle, v, dt)), "V codes/scales differ from the oracle quantiser"
    # K: the device's own fp32 post-norm/RoPE values (rows 0..7 of q_out) through the oracle quantiser
    assert np.array_equal(ks, make_slots(oracle, qo[:, :8], dt)), "K codes/scales differ from the oracle quantiser"


def test_append_yarn_stride_jump(cuda, oracle):
    n = 6
    q = oracle.fill_normal((n, 64, 128), SEED, 41)
    k = oracle.fill_normal((n, 8, 128), SEED, 42)
    v = oracle.fill_normal((n, 8, 128), SEED, 43)
    w = np.ones(128, np.float32)
    inv, af = oracle.rope_table(yarn=1, factor=4.0)
    pos = [0, 39, 40, 41, 500, 3000]
    qo, _, _, _ = run_append(cuda, oracle, "int8", 1e-5, q, k, v, w, w, pos, table=(inv, af), probes=(7, 300000, 40))
    for i, p in enumerate(pos):
        oq, _ = oracle.qk_norm_rope(q[i], k[i], w, w, 1e-5, p, inv, af, 7, 300000, 40)
        assert (np.abs(qo[i] - oq) <= 2e-5 * np.maximum(1.0, np.abs(oq))).all()


@pytest.mark.parametrize("int4", [False, True])
def test_quantiser_bit_exact_vs_reference_cuda_kernels(cuda, oracle, int4):
    """The reference's own kv_quantize_int8/int4_kernel (hy3_gpu.cu:250/:329), run on this GPU."""
    rg = oracle.ref_gpu()
    if rg is None:
        pytest.skip("oracle/_ref/libhy3ref_gpu.so not present")
    dt = "int4" if int4 else "int8"
    n = 24
    k = oracle.fill_normal((n, 8, 128), SEED, 21)
    v = oracle.fill_normal((n, 8, 128), SEED, 22)
    k[0] = 0.0
    v[1, 0] = (np.arange(128, dtype=np.float32) - 64.0) * 0.5
    v[2] *= 1e-6
    v[3] = -7.0
    q = np.zeros((n, 64, 128), np.float32)
    q[:, :8] = k
    w = (1.0 + 0.02 * oracle.fill_normal((128,), SEED, 23)).astype(np.float32)
    inv, af = oracle.rope_table()
    pos = list(range(4090, 4090 + n))
    qo, _, ks, vs = run_append(cuda, oracle, dt, 1e-5, q, k, v, w, w, pos)
    # reference pipeline on the same inputs: its fused norm+rope kernel, then its quantiser
    ref_k = np.stack([rg.qk_norm_rope(q[i], k[i], w, w, pos[i], inv, af)[1] for i in range(n)])
    rks, rvs = rg.kv_quantize(ref_k, v, int4=int4)
    assert np.array_equal(vs, rvs), "V slots differ from the reference CUDA quantiser"
    assert np.array_equal(make_slots(oracle, v, dt), rvs), "oracle quantiser differs from the reference CUDA quantiser"
    # K: feed the reference quantiser the device's own fp32 K -> must be bit-equal to our cache
    rks2, _ = rg.kv_quantize(qo[:, :8], v, int4=int4)
    assert np.array_equal(ks, rks2), "K slots differ from the reference CUDA quantiser on identical fp32 input"
    # end to end (their norm+rope -> their quantiser) vs ours: report, allow +-1 code on rare ulp differences
    same_fp32 = np.array_equal(ref_k, qo[:, :8])
    diff = (rks != ks)
    print("norm+rope fp32 bit-identical to the reference kernel:", same_fp32, "| differing K slot bytes:", int(diff.sum()))
    assert diff.mean() < 0.01


def test_committed_gpu_fixture(cuda, oracle):
    path = os.path.join(ROOT, "tests", "golden", "ref_gpu.npz")
    if not os.path.exists(path):
        pytest.skip("tests/golden/ref_gpu.npz not generated yet")
    g = np.load(path)
    k, v = g["in_k"], g["in_v"]
    n = k.shape[0]
    q = np.zeros((n, 64, 128), np.float32)
    w = np.ones(128, np.float32)
    for dt in ("int8", "int4"):
        _, _, _, vs = run_append(cuda, oracle, dt, 1e-5, q, k, v, w, w, list(range(n)))
        assert np.array_equal(vs, g["vslots_" + dt])
        assert np.array_equal(make_slots(oracle, v, dt), g["vslots_" + dt])
        assert np.array_equal(make_slots(oracle, k, dt), g["kslots_" + dt])
    # the reference's own fused norm + RoPE kernel (hy3_gpu.cu:144-164), run on a B200 when the fixture was made, on the
    # same seeded inputs: the queries must agree bit for bit; K rows take the query path with the K weights for the same check
    q1 = oracle.fill_normal((1, 64, 128), SEED, 1)
    k1 = oracle.fill_normal((1, 8, 128), SEED, 2)
    w2 = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    inv, af = oracle.rope_table()
    inv4, af4 = oracle.rope_table(yarn=1, factor=4.0)
    cases = {"p0": ((inv, af), 0, (1, 0, 0)), "p4096": ((inv, af), 4096, (1, 0, 0)),
             "yarn4_p1048575": ((inv4, af4), 1048575, (1, 0, 0)), "stride7_p300": ((inv, af), 300, (7, 0, 0)),
             "jump_p50": ((inv, af), 50, (1, 300000, 40))}
    for name, (table, pos, probes) in cases.items():
        qo, _, _, _ = run_append(cuda, oracle, "int8", 1e-5, q1, k1, k1, w2[0], w2[1], [pos], table=table, probes=probes)
        assert np.array_equal(qo[0], g["gpu_normrope_%s_q" % name]), "%s: queries differ from the reference CUDA kernel" % name
        qk = np.zeros((1, 64, 128), np.float32)
        qk[0, :8] = k1[0]
        ko, _, _, _ = run_append(cuda, oracle, "int8", 1e-5, qk, k1, k1, w2[1], w2[1], [pos], table=table, probes=probes)
        assert np.array_equal(ko[0, :8], g["gpu_normrope_%s_k" % name]), "%s: keys differ from the reference CUDA kernel" % name


@pytest.mark.parametrize("heads", [(0, 8), (4, 4)])
@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_chunk_kernel_equals_row_kernel(cuda, oracle, dt, heads):
    """Batches of 32 rows or more take the throughput-shaped kernel (one block per row for the queries, one block per KV
    head and 8 rows for K/V); smaller ones the per-row kernel.  Same rows, same slots and positions: identical cache
    bytes and identical fp32 / fp16 queries -- also on a context that owns only KV heads 4..7."""
    import torch
    from hy3_b200 import Hy3Attn
    n, slot0 = 197, 3                         # not a multiple of 8, not aligned: the ragged last K/V block is covered
    q = oracle.fill_normal((n, 64, 128), SEED, 801)
    k = oracle.fill_normal((n, 8, 128), SEED, 802)
    v = oracle.fill_normal((n, 8, 128), SEED, 803)
    w = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    pos = [slot0 + i + (1000 if i > 100 else 0) for i in range(n)]     # RoPE positions need not be the slots
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    res = []
    for step in (n, 16):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=n, max_tokens=512, kv_head_begin=heads[0], kv_head_count=heads[1])
        ctx.set_norm_weights(0, w[0], w[1])
        qo = torch.empty((n, 64, 128), device=cuda)
        q16 = torch.empty((n, 64, 128), dtype=torch.float16, device=cuda)
        for b in range(0, n, step):
            e = min(n, b + step)
            ctx.batch_set([0] * (e - b), list(range(slot0 + b, slot0 + e)), pos[b:e])
            ctx.append(0, tq[b:e], tk[b:e], tv[b:e], q_out=qo[b:e], q_out16=q16[b:e])
        ctx.sync()
        ks, vs = ctx.export_kv(0, 0, slot0, n)
        res.append((qo.cpu().numpy(), q16.cpu().numpy(), ks, vs))
        ctx.close()
    for a, b, what in zip(res[0], res[1], ("q fp32", "q fp16", "K slots", "V slots")):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("seqs", [1, 2])
@pytest.mark.parametrize("heads", [(0, 8), (3, 5), (7, 1)])
@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_chunk_kernel_aligned_columns(cuda, oracle, dt, heads, seqs):
    """The chunk kernel's staged stores (8 aligned consecutive slots; pages crossed; a ragged tail; one KV head per block) and
    a batch of two sequences that must not take them, against the per-row kernel: identical bytes."""
    import torch
    from hy3_b200 import Hy3Attn
    n, slot0 = 75, 104
    q = oracle.fill_normal((n, 64, 128), SEED, 811)
    k = oracle.fill_normal((n, 8, 128), SEED, 812)
    v = oracle.fill_normal((n, 8, 128), SEED, 813)
    v[5] = 0.0
    sid = [0] * n if seqs == 1 else [i % 2 for i in range(n)]
    slots = [slot0 + (i if seqs == 1 else i // 2) for i in range(n)]
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    res = []
    for step in (n, 25):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=2, max_batch=n, max_tokens=1024, max_tokens_per_seq=512, kv_head_begin=heads[0], kv_head_count=heads[1])
        qo = torch.empty((n, 64, 128), device=cuda)
        for b in range(0, n, step):
            e = min(n, b + step)
            ctx.batch_set(sid[b:e], slots[b:e], [3 * x for x in slots[b:e]])
            ctx.append(0, tq[b:e], tk[b:e], tv[b:e], q_out=qo[b:e])
        ctx.sync()
        out = [qo.cpu().numpy()]
        for s in range(seqs):
            out += list(ctx.export_kv(0, s, slot0, sid.count(s)))
        res.append(out)
        ctx.close()
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [8, 40])
@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_rows_without_a_slot_store_nothing(cuda, oracle, dt, n):
    """Rows with slot -1 (no keys in this context) among live ones, in both kernels: their queries come out as usual, no cache byte
    changes but those of the live rows, and the running V scale is the live rows'."""
    import torch
    from hy3_b200 import Hy3Attn
    q = oracle.fill_normal((n, 64, 128), SEED, 821)
    k = oracle.fill_normal((n, 8, 128), SEED, 822)
    v = oracle.fill_normal((n, 8, 128), SEED, 823)
    dead = np.arange(n) % 3 != 1
    v[dead] *= 1e4
    sid = [i % 4 for i in range(n)]                          # every sequence has rows of both kinds
    slots = [-1 if dead[i] else 120 + i for i in range(n)]
    tq, tk, tv = (torch.from_numpy(a).to(cuda) for a in (q, k, v))
    res = []
    for keep in (np.arange(n), np.flatnonzero(~dead)):
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_seqs=4, max_batch=n, max_tokens=4 * 256, max_tokens_per_seq=256)
        for s_ in range(4):
            ctx.fill_random(0, s_, 0, 256, 30 + s_)
        ctx.batch_set([sid[i] for i in keep], [slots[i] for i in keep], list(keep))
        idx = torch.from_numpy(keep).to(cuda)
        qo = ctx.append(0, tq[idx], tk[idx], tv[idx])
        out = ctx.decode(0, qo)
        ctx.sync()
        live = torch.from_numpy(~dead[keep]).to(cuda)
        res.append([qo[live].cpu().numpy(), out[live].cpu().numpy()] + [a for s_ in range(4) for a in ctx.export_kv(0, s_, 0, 256)])
        if len(keep) == n:
            assert not out[~live].any()
            ctx.batch_set([0] * n, [0] * n, list(range(n)))   # the queries of all rows, from a batch without dead ones
            assert torch.equal(ctx.append(0, tq, None, None), qo)
        ctx.close()
    for what, a, b in zip(["queries", "outputs"] + ["cache"] * 8, *res):
        assert np.array_equal(a, b) if what != "outputs" else np.abs(a - b).max() < 1e-3, what


@pytest.mark.parametrize("slot0", [8, 3])
@pytest.mark.parametrize("n,heads", [(1203, (0, 8)), (1203, (3, 5)), (601, (0, 8))])
@pytest.mark.parametrize("dt", ["int8", "int4", "fp16"])
def test_chunk_kernel_head_groups(cuda, oracle, dt, n, heads, slot0, monkeypatch):
    """Chunks long enough for several KV heads per block (groups of 4 + 4, 4 + 1 and 2 x 4 on 148 SMs), with and without aligned
    slots, a ragged tail: identical cache bytes and queries to the per-row kernel; and the prefill operands that the chunk kernel
    writes through give the same attention bits as operands rebuilt from the pages."""
    import torch
    from hy3_b200 import Hy3Attn
    ntok = slot0 + n
    q = torch.from_numpy(oracle.fill_normal((ntok, 64, 128), SEED, 831)).to(cuda)
    k = torch.from_numpy(oracle.fill_normal((ntok, 8, 128), SEED, 832)).to(cuda)
    v = torch.from_numpy(oracle.fill_normal((ntok, 8, 128), SEED, 833)).to(cuda)
    w = (1.0 + 0.02 * oracle.fill_normal((2, 128), SEED, 3)).astype(np.float32)
    res = []
    for step, mirror_mb in ((n, "8192"), (25, "0")):
        monkeypatch.setenv("HY3A_PF_MIRROR_MB", mirror_mb)
        ctx = Hy3Attn(kv_dtype=dt, n_layers=1, max_batch=n, max_tokens=ntok + 128, kv_head_begin=heads[0], kv_head_count=heads[1])
        ctx.set_norm_weights(0, w[0], w[1])
        q16 = torch.empty((ntok, 64, 128), dtype=torch.float16, device=cuda)
        for b, e in [(0, slot0)] + [(b, min(ntok, b + step)) for b in range(slot0, ntok, step)]:
            ctx.batch_set([0] * (e - b), list(range(b, e)))
            ctx.append(0, q[b:e], k[b:e], v[b:e], q_out=False, q_out16=q16[b:e])
        out = ctx.prefill(0, 0, slot0, q16[slot0:])
        ctx.sync()
        res.append([q16.cpu().numpy(), out.cpu().numpy()] + list(ctx.export_kv(0, 0, 0, ntok)))
        ctx.close()
    for what, a, b in zip(("queries", "attention", "K slots", "V slots"), *res):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("n", [2, 31, 32, 33, 336, 337, 600])
def test_batch_descriptor_forms(cuda, oracle, n):
    """The batch descriptor reaches the device as a row range, by value (up to 32 or 336 rows) or as a copy: the same tokens as a
    range and in a shuffled order give the same cache and the same queries, with batches of other forms in between."""
    import torch
    from hy3_b200 import Hy3Attn
    q, k, v = (torch.from_numpy(oracle.fill_normal((n, h, 128), SEED, 700 + h)).to(cuda) for h in (64, 8, 9))
    v = v[:, :8]
    perm = np.random.default_rng(n).permutation(n)
    got = []
    for order in (np.arange(n), perm):
        ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_seqs=2, max_batch=max(n, 40), max_tokens=n + 512, max_tokens_per_seq=n + 128)
        ctx.batch_set([1] * 3, [5, 4, 9])
        ctx.batch_set([0] * n, order, 3 * order if n % 2 else None)
        idx = torch.from_numpy(np.asarray(order)).to(cuda)
        qo = ctx.append(0, q[idx], k[idx], v[idx])
        ctx.batch_set([1], [0])
        ctx.sync()
        back = torch.empty_like(qo)
        back[idx] = qo
        got.append((back, ctx.export_kv(0, 0, 0, n)))
        ctx.close()
    assert torch.equal(got[0][0], got[1][0])
    assert all(np.array_equal(a, b) for a, b in zip(got[0][1], got[1][1]))


def test_launch_count_includes_the_descriptor_kernel(cuda):
    """Every kernel counts: the one that carries a descriptor as well; a descriptor that is copied is none."""
    from hy3_b200 import Hy3Attn
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_batch=400, max_tokens=512)
    for n in (1, 400):
        before = ctx.launches
        ctx.batch_set([0] * n, list(range(n)))
        ctx.append(0, *(torch_rows(cuda, n, h) for h in (64, 8, 8)))
        assert ctx.launches - before == 2
    before = ctx.launches
    ctx.batch_set([0] * 400, list(range(399, -1, -1)))
    assert ctx.launches == before
    ctx.sync()
    ctx.close()


@pytest.mark.parametrize("kv", ["int8", "fp16"])
def test_descriptor_of_a_replayed_step_is_copied(cuda, kv):
    """The descriptor of a step that only a graph reads travels as a copy (no kernel counts), that of an eager one as a kernel, and the
    steps may alternate: without waiting between them and with a synchronisation after every call, the same outputs."""
    import torch
    from hy3_b200 import Hy3Attn
    q, k, v = (torch_rows(cuda, 3, h, 9) for h in (64, 8, 8))
    res = []
    for wait in (False, True):
        ctx = Hy3Attn(kv_dtype=kv, n_layers=2, max_seqs=3, max_batch=3, max_tokens=9000, max_tokens_per_seq=3000)
        for layer in range(2):
            for i in range(3):
                ctx.fill_random(layer, i, 0, 2000, 10 * layer + i)
        out, g_out = torch.zeros((24, 3, 64, 128), device=cuda), torch.zeros((3, 64, 128), device=cuda)
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        ctx.batch_set([0, 1, 2], [99, 5, 700])
        ctx.decode_step(0, q, k, v, out=g_out)
        torch.cuda.synchronize()
        ctx.set_stream(side)
        with torch.cuda.graph(graph, stream=side):
            ctx.decode_step(0, q, k, v, out=g_out)
        ctx.use_torch_stream()
        kernels = []
        for t in range(24):
            before = ctx.launches
            ctx.batch_set([0, 1, 2], [100 + 50 * t, 1999 - 30 * t, 64 * (t % 5)])
            kernels.append(ctx.launches - before)
            if t % 6 == 4:
                ctx.decode_step(1, q, k, v, out=out[t])
            else:
                graph.replay()
                out[t].copy_(g_out)
            if wait:
                torch.cuda.synchronize()
        ctx.sync()
        assert kernels == [int(t % 6 == 5 or t == 0) for t in range(24)]
        res.append(out)
        del graph
        ctx.close()
    assert torch.equal(res[0], res[1])


@pytest.mark.parametrize("kv", ["int8", "fp16"])
def test_batch_descriptor_is_not_overtaken(cuda, kv):
    """Steps enqueued without waiting: every launch reads its own step's descriptor (the next one is written by a kernel that may
    start before the last layer has ended).  Against the same steps with a synchronisation after every call."""
    import torch
    from hy3_b200 import Hy3Attn
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)
    steps, B = 40, 3
    q, k, v = (torch.randn((steps, B, h, 128), device=cuda, generator=gen) for h in (64, 8, 8))
    res = []
    for wait in (False, True):
        ctx = Hy3Attn(kv_dtype=kv, n_layers=2, max_seqs=B, max_batch=48, max_tokens=9000, max_tokens_per_seq=3000)
        for layer in range(2):
            for i in range(B):
                ctx.fill_random(layer, i, 0, 2000, 10 * layer + i)
        out = torch.zeros((steps, 2, B, 64, 128), device=cuda)
        pre = torch.zeros((steps, 40, 64, 128), device=cuda)
        q16 = torch.zeros((40, 64, 128), device=cuda, dtype=torch.float16)
        torch.cuda.synchronize()
        for t in range(steps):
            lens = [100 + 40 * t, 1500 - 30 * t, 7 * t]
            ctx.batch_set(np.arange(B), np.array(lens))
            for layer in range(2):
                ctx.decode_step(layer, q[t], k[t], v[t], out=out[t, layer])
                if wait:
                    ctx.sync()
            if t % 4 == 0:      # a chunk on the first sequence, through the chunk kernel
                m = 40
                ctx.batch_set([0] * m, list(range(lens[0], lens[0] + m)))
                ctx.append(0, q[:m, 0], k[:m, 0], v[:m, 0], q_out=False, q_out16=q16)
                ctx.prefill(0, 0, lens[0], q16, out=pre[t])
                if wait:
                    ctx.sync()
        ctx.sync()
        res.append((out, pre))
        ctx.close()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("kv", ["int8", "fp16", "int4"])
def test_captured_step_leaves_the_descriptor_to_the_next(cuda, kv):
    """A step captured between a batch descriptor and an eager step does not run, so the eager step is the one that has to wait for the
    descriptor: work queued in front keeps all of it in flight.  Then the graph, which must follow the descriptors set before each
    replay, and a capture that holds the descriptor itself.  Against the same steps with a synchronisation after every call."""
    import torch
    from hy3_b200 import Hy3Attn
    gen = torch.Generator(device=cuda)
    gen.manual_seed(4)
    lens = [1500, 40, 700]
    q, k, v = (torch.randn((3, h, 128), device=cuda, generator=gen) for h in (64, 8, 8))
    res = []
    for wait in (False, True):
        ctx = Hy3Attn(kv_dtype=kv, n_layers=2, max_seqs=3, max_batch=3, max_tokens=9000, max_tokens_per_seq=3000)
        for layer in range(2):
            for i in range(3):
                ctx.fill_random(layer, i, 0, 2000, 10 * layer + i)
        out = torch.zeros((8, 3, 64, 128), device=cuda)
        g_out = torch.zeros((3, 64, 128), device=cuda)
        torch.cuda.synchronize()
        side, kept = torch.cuda.Stream(), []
        ctx.set_stream(side)

        def done():
            if wait:
                side.synchronize()

        with torch.cuda.stream(side):
            for t in range(2):
                torch.cuda._sleep(20000000)
                ctx.batch_set([0, 1, 2], [n - 7 * t for n in lens])
                done()
                graph = torch.cuda.CUDAGraph()
                kept.append(graph)
                graph.capture_begin(capture_error_mode="thread_local")
                ctx.decode_step(0, q, k, v, out=g_out)
                graph.capture_end()
                ctx.decode_step(1, q, k, v, out=out[4 * t])
                done()
                ctx.batch_set([0, 1, 2], [n + 9 + t for n in lens])
                done()
                graph.replay()
                done()
                out[4 * t + 1].copy_(g_out)
                done()
                own = torch.cuda.CUDAGraph()
                kept.append(own)
                own.capture_begin(capture_error_mode="thread_local")
                ctx.batch_set([0, 1, 2], [30 + n for n in lens])
                ctx.decode_step(0, q, k, v, out=g_out)
                ctx.decode_step(1, q, k, v, out=out[4 * t + 2])
                own.capture_end()
                own.replay()
                done()
                out[4 * t + 3].copy_(g_out)
                done()
        side.synchronize()
        ctx.use_torch_stream()
        ctx.sync()
        res.append(out)
        del graph, own, kept
        ctx.close()
    assert torch.equal(res[0], res[1])


def test_calls_with_another_device_current(cuda):
    """batch_set launches a kernel: with another device current it goes to the context's device where the stream names it, and is refused
    on a default stream; the prefill's cluster query answers for the context's device; prefill is refused as append and decode are.
    (Two GPUs: skipped where the box has one.)"""
    import torch
    from hy3_b200 import Hy3Attn, Hy3AttnError
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    ctx = Hy3Attn(kv_dtype="int8", n_layers=1, max_batch=64, max_tokens=1024, device=0)
    ctx.fill_random(0, 0, 0, 600, 3)
    q16 = torch.randn((45, 64, 128), device="cuda:0").half()
    q = torch.randn((1, 64, 128), device="cuda:0")
    ctx.sync()
    with torch.cuda.device(1):
        with pytest.raises(Hy3AttnError):
            ctx.batch_set([0], [500])
        cluster = ctx.prefill_cluster(500, 45)
        with pytest.raises(Hy3AttnError):
            ctx.prefill(0, 0, 500, q16, out=torch.zeros((45, 64, 128), device="cuda:0"))
        side = torch.cuda.Stream(device=0)
        ctx.set_stream(side)
        ctx.batch_set([0], [500])
        assert torch.cuda.current_device() == 1
    assert cluster == ctx.prefill_cluster(500, 45) > 1
    with torch.cuda.stream(side):
        got = ctx.decode(0, q)
    side.synchronize()
    ctx.use_torch_stream()
    ctx.batch_set([0], [500])
    want = ctx.decode(0, q)
    ctx.prefill(0, 0, 500, q16)
    ctx.sync()
    assert torch.equal(got, want)
    ctx.close()
