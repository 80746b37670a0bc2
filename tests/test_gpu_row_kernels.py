"""Edges of the kernels that a call's shape selects: remainders of row blocks and tiles, runs of attention splits, chunks of the
state scan, step graphs of many shapes, page edges of the state blob.  References: the same rows one at a time, the
pass kernels (SL_FLAG_PASS_KERNELS, same bits by contract), and the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

from conftest import MINI, TINY, f16_report, gpu_engine
from test_gpu_engine import prompt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines():
    import qwisp_b200 as Q
    args = dict(max_rows=512, kv_pages=512)
    a, b = gpu_engine(MINI, **args), gpu_engine(MINI, flags=Q._lib.SL_FLAG_PASS_KERNELS, **args)
    yield a, b
    a.close(); b.close()


def same(x, y):
    return np.array_equal(np.asarray(x).view(np.uint16), np.asarray(y).view(np.uint16))


# passes of 8, the split form, blocks of 8 / 16 / 32 rows, halves of K, a single tile, rows that fill no block
@pytest.mark.parametrize("M,K,N", [(7, 4096, 6144), (7, 4096, 8192), (3, 2048, 16384), (9, 256, 16), (16, 2048, 2064), (17, 512, 1040), (24, 4096, 48), (33, 4096, 2048),
                                   (64, 2048, 12352), (65, 1024, 4096), (200, 4096, 256), (1200, 256, 32)])
def test_qmm4_row_blocks(M, K, N):
    import torch
    import qwisp_b200 as Q
    from oracle import oracle as O
    L = Q.lib()
    packed, scales, biases = O.synth_q4(3, f"rows.w.{N}.{K}", N, K)
    x = O.synth_f16(3, f"rows.x.{M}.{K}", M * K, 0.0, 1.0).reshape(M, K)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    dw, ds, db, dx = dev(packed), dev(scales), dev(biases), dev(x)
    wr = torch.empty((N // 16) * (K // 128) * 1024, dtype=torch.uint8, device="cuda")
    sr = torch.empty((N // 16) * (K // 128) * 128, dtype=torch.uint8, device="cuda")
    assert L.sl_op_repack_q4_device(ptr(dw), ptr(ds), ptr(db), K, N, ptr(wr), ptr(sr), None) == 0
    y = torch.zeros(M * N, dtype=torch.float16, device="cuda")
    one = torch.zeros(M * N, dtype=torch.float16, device="cuda")
    assert L.sl_op_qmm4_device(ptr(dx), ptr(wr), ptr(sr), M, K, N, ptr(y), None) == 0
    for m in range(M):
        assert L.sl_op_qmm4_device(C.c_void_p(dx.data_ptr() + m * K * 2), ptr(wr), ptr(sr), 1, K, N, C.c_void_p(one.data_ptr() + m * N * 2), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int16), one.view(torch.int16))
    if K % 512:
        return                                        # (the oracle walks blocks of 512 inputs)
    few = [0, M // 2, M - 1]
    assert f16_report(y.cpu().numpy().reshape(M, N)[few], O.qmm4(np.ascontiguousarray(x[few]), packed, scales, biases))["max_abs"] <= 2e-2


# rows of one stream behind nothing, behind one 32-key split and behind more splits than a CTA's run
@pytest.mark.parametrize("base", [0, 33, 1100])
@pytest.mark.parametrize("M", [2, 8, 16, 24, 25, 32, 33, 64, 131])
def test_rows_of_one_stream(engines, base, M):
    V = MINI["vocab"]
    toks = prompt(V, base + M + 1, f"rowk.{base}.{M}")
    out = []
    for e in engines:
        s = e.stream(base + M + 8)
        for i in range(0, base, 300):
            s.forward(toks[i:min(i + 300, base)], want_hidden=False)
        out.append((s.step_logits(toks[base:base + M]), s.step_argmax(toks[base + M:]), s.state_save()))
        assert not e.gpu_fault()
        s.close()
    (la, ta, ba), (lb, tb, bb) = out
    assert same(la, lb) and np.array_equal(ta, tb) and np.array_equal(ba, bb)


# rows that the expert kernels route for themselves (up to 24) and one more; experts of one block and of several
@pytest.mark.parametrize("M", [2, 8, 9, 23, 24, 25])
def test_rows_routed_by_the_expert_kernels(engines, M):
    import qwisp_b200 as Q
    toks = prompt(MINI["vocab"], 3 + M, f"route.{M}")
    x = np.random.default_rng(M).standard_normal((M, MINI["hidden"])).astype(np.float16)
    out = []
    for e in engines:
        s = e.stream(M + 8)
        s.forward(toks[:3], want_hidden=False)
        out.append((s.forward(toks[3:]), s.state_save()) + tuple(Q.ops.moe_block(e, 0, x)))
        s.close()
    (ha, ba, oa, ia, sa), (hb, bb, ob, ib, sb) = out
    assert same(ha, hb) and np.array_equal(ba, bb) and same(oa, ob) and np.array_equal(ia, ib) and same(sa, sb)


# expert blocks of 16 rows (a mean of more than 8 rows an expert): blocks of at most 8 rows among them, one and many blocks of an expert
@pytest.mark.parametrize("M", [25, 30, 47, 66, 257, 512])
def test_expert_blocks_of_sixteen_rows(engines, M):
    import qwisp_b200 as Q
    x = np.random.default_rng(M).standard_normal((M, MINI["hidden"])).astype(np.float16)
    (oa, ia, sa), (ob, ib, sb) = (Q.ops.moe_block(e, 0, x) for e in engines)
    counts = np.bincount(ia.ravel(), minlength=MINI["n_experts"])
    assert M * MINI["top_k"] > 8 * MINI["n_experts"] and np.any(counts > 8) and np.any((counts - 1) % 16 < 8)
    assert np.array_equal(ia, ib) and same(sa, sb) and same(oa, ob)


# chunks of the state scan: a chunk less or more one row, remainders of its turns, behind a history
@pytest.mark.parametrize("M", [3, 5, 47, 48, 49, 50, 97, 145])
def test_state_scan_chunks(engines, M):
    V = MINI["vocab"]
    toks = prompt(V, 5 + M, f"scan.{M}")
    out = []
    for e in engines:
        s = e.stream(M + 8)
        s.forward(toks[:5], want_hidden=False)
        out.append((s.forward(toks[5:]), s.state_save()))
        s.close()
    assert same(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


# streams of very different lengths in one step: the one-row form of the state update, the two-kernel form, one wave of attention and more
@pytest.mark.parametrize("B", [2, 5, 6, 9, 17, 23])
def test_batches_of_ragged_streams(engines, B):
    V = MINI["vocab"]
    a = engines[0]
    lens = [1 + (i * 37) % 90 + (700 if i == 1 else 0) for i in range(B)]
    solo, lane, cur = [], [], []
    for i, n in enumerate(lens):
        p = prompt(V, n, f"ragged.{i}")
        for group in (solo, lane):
            s = a.stream(n + 8)
            for j in range(0, n, 300):
                t = s.step_argmax(p[j:j + 300])
            group.append(s)
        cur.append(int(t[-1]))
    cur_lane = list(cur)
    for _ in range(2):
        cur = [int(s.step_argmax([t])[0]) for s, t in zip(solo, cur)]
        cur_lane = [int(t) for t in a.batch_step_argmax(lane, cur_lane)]
        assert cur == cur_lane
    for x, y in zip(solo, lane):
        assert np.array_equal(x.state_save(), y.state_save())
        x.close(); y.close()


# token tiles and weight-row groups of the tensor-core product; runs of several items in which a warp's second tile comes and goes
@pytest.mark.parametrize("M,K,N", [(1, 512, 16), (31, 512, 128), (33, 512, 144), (65, 1024, 2064), (129, 4096, 272), (1000, 512, 144), (20000, 512, 144), (6000, 512, 1040)])
def test_tensor_core_tiles(M, K, N):
    from test_gpu_ops import test_tensor_core_gemm_matches_gemv_and_oracle as check
    check(M, K, N)


# expert blocks of 32, 48 and 64 rows (means of 20, 21, 34, 35 rows an expert and others) in prefill mode: the same rows in one call
@pytest.mark.parametrize("cuts", [[41, 42], [69, 70], [1, 61, 130], [300, 42]])
def test_prefill_expert_blocks(engines, cuts):
    e = engines[0]
    toks = prompt(MINI["vocab"], sum(cuts), "blocks")
    a, b = e.stream(400), e.stream(400)
    whole = a.forward_hybrid(toks)
    parts = np.concatenate([b.forward_hybrid(toks[sum(cuts[:i]):sum(cuts[:i + 1])]) for i in range(len(cuts))])
    assert same(whole, parts) and np.array_equal(a.state_save(), b.state_save())
    a.close(); b.close()


# vocabularies of less than a strand, of a remainder in the last CTA, of many rounds, and of more logits than shared memory holds
@pytest.mark.parametrize("vocab", [16, 1040, 20496, 431104])
def test_sampler_vocabularies(vocab):
    import qwisp_b200 as Q
    from oracle import oracle as O
    e = gpu_engine(dict(TINY, vocab=vocab, n_layers=2), max_streams=1, max_rows=4)
    try:
        logits = O.synth_f16(7, "vocab.logits", 3 * vocab, 0.0, 2.5).reshape(3, vocab)
        adj = O.synth_f16(7, "vocab.adj", vocab, 0.0, 0.5).astype(np.float32)
        logits[1, :] = logits[1, 0]                               # a tie of all
        logits[2, vocab - 3] = np.float16(-np.inf)
        draft = np.array([int(np.argmax(logits[0].astype(np.float32))), vocab - 1, -1], dtype=np.int32)
        for inv_t, top_p, a in ((0.0, 1.0, None), (1.0 / 0.7, 1.0, adj), (1.0, 0.9, None), (1.0 / 0.7, 0.95, adj)):
            got = Q.ops.sample_rows(e, logits, draft, inv_t, top_p, 5, 6, 40, logit_adj=a)
            ref = O.sample_rows(logits, draft, inv_t, top_p, 5, 6, 40, logit_adj=a)
            assert all(np.array_equal(g, r) for g, r in zip(got, ref)), (inv_t, top_p, got, ref)
    finally:
        e.close()


# so many likely tokens that the histogram's counts wrap, and their sums pass the target (0.9 of what is left of the total) in two bins
def test_sampler_counts_wrap():
    import qwisp_b200 as Q
    from oracle import oracle as O
    parts = ((366000, 0.0), (169200, -0.0625), (92800, -3.921875))          # tokens, logit: bins 0, 1 and 100
    sums = np.cumsum([n * int(np.exp(np.float32(x)) * 8192) for n, x in parts]) % 2 ** 32
    assert sums[0] > 0.9 * sums[2] > sums[1] and sum(n for n, _ in parts) % 16 == 0
    row = np.concatenate([np.full(n, x, np.float16) for n, x in parts])
    e = gpu_engine(dict(TINY, vocab=row.size, n_layers=2), max_streams=1, max_rows=8)
    try:
        logits = np.stack([np.random.default_rng(i).permutation(row) for i in range(8)])
        draft = np.full(8, -1, dtype=np.int32)
        for pos in range(0, 160, 8):
            got = Q.ops.sample_rows(e, logits, draft, 1.0, 0.9, 5, 6, pos)
            ref = O.sample_rows(logits, draft, 1.0, 0.9, 5, 6, pos)
            assert all(np.array_equal(g, r) for g, r in zip(got, ref)), (pos, got, ref)
            assert all(logits[i, t] == 0 for i, t in enumerate(ref[0]))
    finally:
        e.close()


# strict calls of every length that has a step graph, with two heads, some of them again
def test_step_graphs_of_many_shapes():
    import qwisp_b200 as Q
    V = TINY["vocab"]
    a, b = gpu_engine(TINY), gpu_engine(TINY, flags=Q._lib.SL_FLAG_NO_GRAPH)
    try:
        toks = prompt(V, 64, "graphs")
        for rows in list(range(2, 65)) + [64, 3, 2]:
            got = []
            for e in (a, b):
                s = e.stream(160)
                got.append((s.step_argmax(toks[:rows]), s.step_argmax(toks[:2]), s.step_logits(toks[:rows])))
                s.close()
            assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1]) and same(got[0][2], got[1][2]), rows
        assert not a.gpu_fault()
    finally:
        a.close(); b.close()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 250])
def test_state_blob_at_page_edges(engines, n):
    V = MINI["vocab"]
    a, b = engines[0], engines[1]
    s = a.stream(n + 8)
    s.step_argmax(prompt(V, n, f"page.{n}"))
    blob = s.state_save()
    t = b.stream(n + 40)                              # other arena, other pages
    assert t.state_restore(blob) and np.array_equal(t.state_save(), blob)
    assert np.array_equal(s.step_argmax([7, 11]), t.step_argmax([7, 11]))
    assert np.array_equal(s.state_save(), t.state_save())
    s.close(); t.close()


# one vocabulary row gives NaN: it is passed over, and hides no other logit of its 16-row tile (9 rows and more: the many-row head)
@pytest.mark.parametrize("rows", [8, 9, 16, 17, 33])
def test_head_passes_over_nan_logits(tiny_oracle, rows):
    import qwisp_b200 as Q
    V, H = TINY["vocab"], TINY["hidden"]
    tensors = {n: tiny_oracle.tensor_bytes(n).copy() for n in tiny_oracle.tensor_names()}
    cfg = Q.config(**TINY, max_rows=64, max_streams=2, kv_page_size=32, kv_pages=8)
    toks = prompt(V, rows, "nan")
    clean = Q.Engine.from_tensors(cfg, tensors)
    want = clean.stream(64).step_argmax(toks)
    clean.close()
    bad = {int(t) // 16 * 16 for t in want} - {int(t) for t in want}
    assert bad
    biases = tensors["lm_head.b"].view(np.float16).reshape(V, H // 64).copy()
    biases[sorted(bad)] = np.nan
    tensors["lm_head.b"] = biases
    eng = Q.Engine.from_tensors(cfg, tensors)
    got = eng.stream(64).step_argmax(toks)
    eng.close()
    assert np.array_equal(got, want)


# rows whose places pass 2^32 halves (8.6 GB of activations): each row gives what it gives alone
def test_tensor_core_product_of_very_many_rows():
    import torch
    import qwisp_b200 as Q
    from oracle import oracle as O
    L = Q.lib()
    K, N, M = 4096, 16, (1 << 20) + 200
    packed, scales, biases = O.synth_q4(3, "tall.w", N, K)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    dw, ds, db = dev(packed), dev(scales), dev(biases)
    wr = torch.empty((N // 16) * (K // 128) * 1024, dtype=torch.uint8, device="cuda")
    sr = torch.empty((N // 16) * (K // 128) * 128, dtype=torch.uint8, device="cuda")
    assert L.sl_op_repack_q4_device(ptr(dw), ptr(ds), ptr(db), K, N, ptr(wr), ptr(sr), None) == 0
    x = torch.zeros((M, K), dtype=torch.float16, device="cuda")
    few = 300                                         # the rows on both sides of the boundary
    x[M - few:] = torch.randn((few, K), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda").half()
    y = torch.empty((M, N), dtype=torch.float16, device="cuda")
    want = torch.empty((few, N), dtype=torch.float16, device="cuda")
    assert L.sl_op_qmm4_tc_device(ptr(x), ptr(wr), ptr(sr), M, K, N, ptr(y), None) == 0
    assert L.sl_op_qmm4_tc_device(ptr(x[M - few:]), ptr(wr), ptr(sr), few, K, N, ptr(want), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(y[M - few:].view(torch.int16), want.view(torch.int16)) and not y[:M - few].any()
