"""Host-side failures and host-side rules of the library, without a GPU: each test runs a child process in which a stand-in for the
CUDA runtime (fake_cudart.cpp) is preloaded, which also stands for NCCL.  It gives memory, runs no kernels, and fails the calls it is told to fail."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT, TINY

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = f"""
import ctypes as C, sys
sys.path.insert(0, {ROOT!r})
import numpy as np
import qwisp_b200 as Q
F = C.CDLL(None)
F.fake_count.restype = C.c_long
F.fake_unpacked.restype = C.c_long
F.fake_fail_alloc.argtypes = [C.c_size_t]
F.fake_fail_threads.argtypes = F.fake_fail_launches.argtypes = [C.c_long]
F.fake_launched.restype = C.c_long
F.fake_launched.argtypes = [C.c_char_p, C.c_uint]
count = lambda what: F.fake_count(what.encode())
GEOM = {TINY!r}

def engine(**kw):
    args = dict(max_rows=128, max_streams=80, kv_page_size=32, kv_pages=1024)
    args.update(kw)
    return Q.Engine.synthetic(Q.config(**GEOM, **args), seed=1)

def refused(code, fn, *a):
    try:
        fn(*a)
    except Q.SeedlessError as e:
        assert e.code == code, e
    else:
        raise AssertionError("the call went through")

def filled(eng, n):
    s = eng.stream(n + 8)
    for i in range(0, n, 128):
        s.forward(list(range(min(128, n - i))), want_hidden=False)
    assert s.length == n
    return s

def blob_of(n):          # a valid blob of n positions, its data words numbered
    gdn = [np.array([2, 3 * 4096, 16 * 128 * 128], dtype=np.uint32), np.zeros(3 * 4096 // 2 + 16 * 128 * 128, dtype=np.uint32)]
    att = [np.array([1, 1, 256, n], dtype=np.uint32), np.zeros(2 * n * 128, dtype=np.uint32)]
    w = np.concatenate([np.array([0x31535751, 1, 4], dtype=np.uint32)] + gdn + att + gdn + att)
    zero = w == 0
    w[zero] = np.arange(w.size, dtype=np.uint32)[zero]
    return w
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", os.path.join(HERE, "fake_cudart.cpp"),
                    "-o", so, "-ldl", "-lpthread"], check=True, timeout=120)
    os.symlink(so, os.path.join(os.path.dirname(so), "libnccl.so.2"))
    env = dict(os.environ, LD_PRELOAD=so, LD_LIBRARY_PATH=os.path.dirname(so) + os.pathsep + os.environ.get("LD_LIBRARY_PATH", ""))

    def run(script):
        out = subprocess.run([sys.executable, "-c", PRELUDE + script], env=env, capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-3000:]
    return run


def test_state_io_without_room_is_refused_and_the_engine_goes_on(fake):
    """The slots of state save and restore cannot be allocated: the call is refused, the stream is as it was, a later call works."""
    fake("""
e = engine()
s = filled(e, 40)
F.fake_fail_alloc(32 << 20)
refused(-5, s.state_save)
assert e.gpu_fault() is None and s.length == 40
assert len(s.step_argmax([1, 2])) == 2 and s.length == 42
F.fake_fail_alloc(0)
blob = s.state_save()
e2 = engine()
t = e2.stream(64)
F.fake_fail_alloc(32 << 20)
good = blob_of(42).view(np.uint8)
assert good.size == blob.size
refused(-5, t.state_restore, good)
assert e2.gpu_fault() is None and t.length == 0
F.fake_fail_alloc(0)
assert t.state_restore(good) and t.length == 42
""")


@pytest.mark.parametrize("n", [1, 1000, 3000, 4088, 16000])
def test_state_io_moves_every_word_and_only_the_calling_thread_calls_cuda(fake, n):
    """A blob of one range, some, and more than there are slots: each word is saved and restored once, and no helper thread makes a
    CUDA call (a host's per-thread stream would be another stream there)."""
    fake(f"n = {n}" + """
e = engine(kv_pages=520)
s = filled(e, n)
blob = s.state_save().view(np.uint32)
assert np.array_equal(blob, np.arange(blob.size, dtype=np.uint32))     # (the stand-in packs each word's number)
t = engine(kv_pages=520).stream(n + 8)
want = blob_of(n)
assert want.size == blob.size and t.state_restore(want.view(np.uint8)) and t.length == n
got = np.zeros_like(want)
assert F.fake_unpacked(got.ctypes.data_as(C.c_void_p), C.c_long(want.size)) == want.size
assert np.array_equal(got, want)
assert count("other_thread") == 0
""")


def test_state_io_reports_a_failed_launch(fake):
    """A pack kernel that cannot be launched is an error of the call, from whichever range on."""
    fake("""
e = engine(kv_pages=520)
s = filled(e, 16000)
F.fake_fail_launches(9)
refused(-3, s.state_save)
assert e.gpu_fault() is not None
F.fake_fail_launches(-1)
refused(-4, s.step_argmax, [1])
""")


@pytest.mark.parametrize("threads", [0, 1, 3])
def test_state_io_without_threads_to_be_had(fake, threads):
    """Thread starts fail from some point on: the threads there are, or the caller alone, do the work."""
    fake(f"threads = {threads}" + """
n = 16000
e = engine(kv_pages=520)
s = filled(e, n)
t = engine(kv_pages=520).stream(n + 8)
before = count("threads")
F.fake_fail_threads(threads)
blob = s.state_save().view(np.uint32)
assert np.array_equal(blob, np.arange(blob.size, dtype=np.uint32)) and count("threads") == before + threads
F.fake_fail_threads(threads)
want = blob_of(n)
assert t.state_restore(want.view(np.uint8))
got = np.zeros_like(want)
assert F.fake_unpacked(got.ctypes.data_as(C.c_void_p), C.c_long(want.size)) == want.size and np.array_equal(got, want)
F.fake_fail_threads(-1)
""")


def test_batched_steps_of_any_size_replay_a_graph(fake):
    """Batches of more than 64 streams are captured at their second step and replayed from then on, like smaller ones."""
    fake("""
e = engine()
streams = [e.stream(32) for _ in range(80)]
for b in (64, 65, 80):
    for k in range(4):
        made, ran = count("graphs_made"), count("graph_launches")
        e.batch_step_argmax(streams[:b], [1] * b)
        assert (count("graphs_made") - made, count("graph_launches") - ran) == [(0, 0), (1, 1), (0, 1), (0, 1)][k], (b, k)
""")


def test_step_graphs_are_made_once_per_shape(fake):
    """Every verify, sampling and forward length of one stream and many batch sizes, round and round: a capture each, no graph dropped."""
    fake("""
e = engine(kv_pages=2000)
s = e.stream(30000)
streams = [e.stream(200) for _ in range(40)]
for turn in range(3):
    made, ran = count("graphs_made"), count("graph_launches")
    for rows in range(2, 65):
        s.step_argmax([1] * rows)
        s.step_logits([1] * rows)
        s.forward([1] * rows)
    for b in range(2, 41):
        e.batch_step_argmax(streams[:b], [1] * b)
    shapes = 3 * 63 + 39
    assert (count("graphs_made") - made, count("graph_launches") - ran) == [(0, 0), (shapes, shapes), (0, shapes)][turn], turn
assert count("graphs_dropped") == 0
""")


def test_calls_on_the_legacy_stream_run_eagerly(fake):
    """A host that handed over cudaStreamLegacy (handle 1), which cannot be captured: calls of every kind go on without graphs."""
    fake("""
e = engine()
e.set_cuda_stream(1)
s = e.stream(200)
streams = [e.stream(32) for _ in range(3)]
for _ in range(3):
    s.forward([1, 2, 3])
    s.step_argmax([1, 2])
    s.step_argmax([1])
    e.batch_step_argmax(streams, [1, 2, 3])
assert count("captures") == 0 and e.gpu_fault() is None
""")


def test_no_room_for_a_graph_is_no_failure(fake):
    """A graph that cannot be made for lack of memory: the call, and later ones of its shape, are launched eagerly."""
    fake("""
e = engine()
s = e.stream(200)
F.fake_fail_graphs(1)
for _ in range(4):
    assert len(s.step_argmax([1, 2, 3])) == 3
assert count("graphs_made") == 0 and count("graph_launches") == 0 and e.gpu_fault() is None
assert count("captures") == 1                                  # (tried once)
F.fake_fail_graphs(0)
for _ in range(3):
    s.step_argmax([1, 2])
assert count("graphs_made") == 1 and count("graph_launches") == 2
""")


def test_every_launch_is_counted(fake):
    """sl_engine_launch_count counts each kernel that a call launches: steps, sampling, prefill, state save and restore, rollback."""
    fake("""
e = engine()
e.use_graphs(False)
s, t = e.stream(200), e.stream(200)
blob = blob_of(40).view(np.uint8)
snap = s.snapshot()
calls = [lambda: s.step_argmax([1]), lambda: s.rollback(snap), lambda: s.step_sample_rows([1, 2], None, 1.0, 0.9, 1, 2, 0), lambda: s.forward_hybrid([1] * 40),
         lambda: s.forward([1] * 40), lambda: s.step_argmax([1, 2]), lambda: e.batch_step_argmax([s, t], [1, 2]), lambda: s.state_save(),
         lambda: t.state_restore(blob), lambda: Q.ops.lm_head(e, np.zeros((3, 512), np.float16))]
for i, call in enumerate(calls):
    ran, counted = count("launches"), e.launch_count()
    call()
    assert count("launches") - ran == e.launch_count() - counted > 0, (i, count("launches") - ran, e.launch_count() - counted)
""")


@pytest.mark.parametrize("rows", [5, 13, 16, 17, 30])
def test_expert_block_height_of_an_expert_parallel_step(fake, rows):
    """Blocks of 8 rows (24 warps and the producer) up to a mean of 8 gathered rows an expert, of 16 rows (16 warps and the producer) from there
    on, as in a plain call of as many rows: the rule goes by the experts of the model, in an expert-parallel step too."""
    fake(f"rows = {rows}" + """
blocks = lambda: [F.fake_launched(b"k_expert_rows", t) for t in (25 * 32, 17 * 32)]
gathered, wide = 2 * rows, 2 * rows * GEOM["top_k"] > 8 * GEOM["n_experts"]
ep = engine()
ep.use_graphs(False)
ep.ep_init(0, 2, np.zeros(128, np.uint8), rows)
streams = [ep.stream(32) for _ in range(rows)]
before = blocks()
assert len(ep.batch_step_argmax(streams, [1] * rows)) == rows and F.fake_launched(b"k_ep_lists", 256) == GEOM["n_layers"]
one = [b - a for a, b in zip(before, blocks())]
assert one == [2 * GEOM["n_layers"] * (not wide), 2 * GEOM["n_layers"] * wide], one
if gathered > 24:                                          # (shorter plain calls are routed by the expert kernels: always 8 rows)
    s, before = ep.stream(128), blocks()
    s.forward([1] * gathered)
    assert [b - a for a, b in zip(before, blocks())] == one
""")
