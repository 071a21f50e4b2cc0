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
