"""Partial sums of matvecs whose columns are split: the room in memory that a stream's launches exchange them through.

The exchange through memory and the one as clusters give the same bits (test_gpu_tensor_core_matvec.py), so what is checked here is which of them a
launch takes, and that streams which overlap do not share a room.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

from vinf_3080ti_b200.gguf_types import GGUFTensorType as T
from vinf_3080ti_b200.synth import synthetic_activations, synthetic_blocks

pytestmark = pytest.mark.gpu
TYPE, ROWS, COLS, M = T.Q4_K, 2305, 2304, 4  # split columns
PER_THREAD = 2  # the handle cudaStreamPerThread
N = 12


class Passes:
    """A runtime with N inputs, N outputs, and what the passes over them have to give."""

    def __init__(self, codebooks):
        from vinf_3080ti_b200.runtime import Runtime

        rng = np.random.default_rng(0)
        self.rt = Runtime(codebooks["iq3s_grid"], codebooks)
        self.rt.upload("w", synthetic_blocks(TYPE, ROWS, COLS, rng), int(TYPE), COLS, ROWS)
        for i in range(N):
            self.rt.alloc(f"x{i}", M * COLS)
            self.rt.alloc(f"y{i}", M * ROWS)
            self.rt.write(f"x{i}", synthetic_activations(M, COLS, rng))
        self.rt.capture_begin()  # (in a capture: clusters)
        for i in range(N):
            self.launch(i)
        graph = self.rt.capture_end()
        self.rt.graph_launch(graph)
        self.rt.synchronize()
        self.rt.graph_destroy(graph)
        self.want = [self.read(i) for i in range(N)]
        assert self.rt.memory_exchange_count() == 0

    def launch(self, i):
        self.rt.qmv("w", f"x{i}", f"y{i}", M)

    def read(self, i):
        return self.rt.read_array(f"y{i}", M * ROWS).copy().view(np.uint32)

    def clear(self):
        for i in range(N):
            self.rt.zero(f"y{i}")
        self.rt.synchronize()

    def exchanged(self, work):
        """What `work` adds to the count of exchanges through memory."""
        before = self.rt.memory_exchange_count()
        work()
        return self.rt.memory_exchange_count() - before

    def check(self):
        self.rt.set_stream(None)
        self.rt.synchronize()
        for i in range(N):
            assert np.array_equal(self.read(i), self.want[i]), i


@pytest.fixture
def two(codebooks):
    """Two runtimes, both of which have launched: the GPU is shared."""
    passes = [Passes(codebooks) for _ in range(2)]
    for p in passes:
        p.launch(0)
        p.rt.synchronize()
        p.clear()
    yield passes
    for p in passes:
        p.rt.close()


def test_a_stream_set_while_it_was_captured_has_a_room_afterwards(two):
    import torch

    p, stream, graph = two[0], torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        p.rt.set_stream(stream.cuda_stream)
        captured = p.exchanged(lambda: p.launch(0))
        graph.capture_end()
    assert captured == 0
    assert p.exchanged(lambda: [p.launch(i) for i in range(1, N)]) == N - 1
    with torch.cuda.stream(stream):
        graph.replay()
    p.check()


def test_threads_on_their_own_default_streams_have_rooms_of_their_own(two):
    p, go_on, counts = two[0], threading.Event(), {}
    p.rt.set_stream(PER_THREAD)

    def passes(first):  # (one thread at a time calls; the first one's stream lives on beside the second's)
        counts[first] = p.exchanged(lambda: [p.launch(i) for _ in range(8) for i in range(first, N, 2)])

    def first():
        passes(0)
        done.set()
        go_on.wait(60)

    done = threading.Event()
    thread = threading.Thread(target=first)
    thread.start()
    assert done.wait(60)
    try:
        passes(1)
        p.rt.synchronize()
    finally:
        go_on.set()
        thread.join()
    assert counts == {0: 8 * N // 2, 1: 8 * N // 2}
    p.check()


def test_closing_a_runtime_of_two_streams_beside_an_open_capture(two):
    import torch

    gone, p = two
    gone.rt.set_stream(torch.cuda.Stream().cuda_stream)
    assert gone.exchanged(lambda: gone.launch(0)) == 1
    opened, closed, failures = threading.Event(), threading.Event(), []

    def capture():
        try:
            p.rt.capture_begin()
            for i in range(N):
                p.launch(i)
            opened.set()
            closed.wait(60)
            graph = p.rt.capture_end()
            p.rt.graph_launch(graph)
            p.rt.synchronize()
            p.rt.graph_destroy(graph)
        except Exception as e:  # noqa: BLE001
            failures.append(e)
        finally:
            opened.set()

    thread = threading.Thread(target=capture)
    thread.start()
    assert opened.wait(60)
    try:
        gone.rt.close()
    finally:
        closed.set()
        thread.join()
    assert not failures
    p.check()


@pytest.mark.parametrize("t,rows,cols,per_launch", [(T.Q6_K, 2305, 2304, 24), (T.Q3_K, 1030, 5120, 16), (T.Q8_0, 4099, 1280, 8)], ids=str)
def test_every_row_count_goes_through_memory_and_gives_what_clusters_give(two, t, rows, cols, per_launch):
    rt = two[0].rt
    rng = np.random.default_rng(rows)
    rt.upload("v", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    rt.alloc("x", 24 * cols)
    rt.alloc("y", 24 * rows)
    for m in (1, 2, 4, 8, 16, 24):
        rt.write("x", synthetic_activations(m, cols, rng))
        rt.zero("y")
        through_memory = two[0].exchanged(lambda: rt.qmv("v", "x", "y", m))
        rt.synchronize()
        assert through_memory == -(-m // per_launch), m
        got = rt.read_array("y", m * rows).copy()
        rt.zero("y")
        rt.capture_begin()
        rt.qmv("v", "x", "y", m)
        graph = rt.capture_end()
        rt.graph_launch(graph)
        rt.synchronize()
        rt.graph_destroy(graph)
        assert np.abs(got).max() > 0 and np.array_equal(got.view(np.uint32), rt.read_array("y", m * rows).view(np.uint32)), m


def test_streams_of_one_runtime_that_overlap(two):
    import torch

    p, streams = two[0], [torch.cuda.Stream() for _ in range(3)]
    for _ in range(5):
        p.clear()
        for stream in streams:
            with torch.cuda.stream(stream):
                torch.cuda._sleep(2_000_000)  # some 1 ms: all launches are there before the first runs
        before = p.rt.memory_exchange_count()
        for i in range(N):
            p.rt.set_stream(streams[i % 3].cuda_stream)
            p.launch(i)
        assert p.rt.memory_exchange_count() - before == N
        p.check()


def test_the_fifth_stream_of_a_runtime_has_clusters(two):
    import torch

    p, streams = two[0], [torch.cuda.Stream() for _ in range(4)]
    for i, stream in enumerate(streams):  # (the first is the runtime's own)
        p.rt.set_stream(stream.cuda_stream)
        assert p.exchanged(lambda: [p.launch(k) for k in range(i, N, 4)]) == (N // 4 if i < 3 else 0)
    p.check()


def test_rooms_run_out_and_come_back(two, codebooks):
    import torch

    p, others = two[0], []
    try:
        while len(others) < 20:
            others.append(Passes(codebooks))
            if others[-1].exchanged(lambda: others[-1].launch(0)) == 0:
                break
        assert 2 <= len(others) < 20  # 16 rooms of a process
        last = others[-1]
        assert last.exchanged(lambda: [last.launch(i) for i in range(N)]) == 0
        last.check()
        last.clear()
        others.pop(0).rt.close()
        assert last.exchanged(lambda: [last.launch(i) for i in range(N)]) == N
        last.check()
    finally:
        for other in others:
            other.rt.close()
    stream = torch.cuda.Stream()
    for _ in range(18):  # whose last work is on a stream of the caller
        gone = Passes(codebooks)
        gone.rt.set_stream(stream.cuda_stream)
        assert gone.exchanged(lambda: gone.launch(0)) == 1
        gone.rt.set_stream(None)
        gone.rt.close()
        p.rt.synchronize()


ALONE = """
import sys
import numpy as np
sys.path.insert(0, {repo!r})
from tests.test_gpu_stream_partials import N, Passes
with np.load({repo!r} + "/tests/golden/iq_codebooks.npz") as z:
    books = {{k: z[k].tobytes() for k in z.files}}
counts = []
def run(p):
    counts.append(p.exchanged(lambda: [p.launch(i) for i in range(N)]))
    p.check()
    p.clear()
first = Passes(books)
run(first)
second = Passes(books)  # (nothing but captured launches yet)
run(first)
run(second)
run(first)
second.rt.close()
run(first)
print(counts)
"""


def test_clusters_while_one_stream_has_the_gpu_to_itself():
    import subprocess
    import sys
    from pathlib import Path

    repo = str(Path(__file__).resolve().parent.parent)
    done = subprocess.run([sys.executable, "-c", ALONE.format(repo=repo)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    assert done.stdout.split("\n")[0] == str([0, 0, N, N, 0])
