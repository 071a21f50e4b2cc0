"""The scratch of passes of more than 8 rows (B operands, partial sums) as a runtime's tensors and streams change."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import dequant_np as O
from vinf_3080ti_b200.gguf_types import GGUFTensorType as T
from vinf_3080ti_b200.synth import synthetic_activations, synthetic_blocks

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5  # as for the tensor-core matvec


@pytest.fixture
def rt(codebooks):
    from vinf_3080ti_b200.runtime import Runtime

    runtime = Runtime(codebooks["iq3s_grid"], codebooks)
    yield runtime
    runtime.close()


def captured(rt, work):
    """`work` as a graph, launched once: in a capture the blocks that share columns are clusters."""
    rt.capture_begin()
    work()
    graph = rt.capture_end()
    rt.graph_launch(graph)
    rt.synchronize()
    rt.graph_destroy(graph)


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K], ids=lambda t: t.name)
def test_scratch_that_has_grown_several_times(rt, codebooks, t):
    rows = 1024
    rng = np.random.default_rng(int(t))
    for cols in (2304, 28928, 38400, 51200):  # each but the first outgrows the scratch, by less than half
        raw = synthetic_blocks(t, rows, cols, rng)
        rt.upload("w", raw, int(t), cols, rows)
        for m in (24, 16, 9):
            x = synthetic_activations(m, cols, rng)
            rt.alloc("x", m * cols)
            rt.alloc("y", m * rows)
            rt.write("x", x)
            outs = []
            for run in (lambda work: work(), lambda work: captured(rt, work)):
                rt.zero("y")
                run(lambda: rt.qmv("w", "x", "y", m))
                rt.synchronize()
                outs.append(rt.read_array("y", m * rows).copy())
            assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32)), (cols, m)
        ref = O.matvec(raw, int(t), rows, cols, x[:1], codebooks)
        got = outs[0].reshape(m, rows)[0]
        assert np.linalg.norm(got - ref[0]) <= REL_L2 * np.linalg.norm(ref[0]), cols


def test_a_stream_on_which_the_scratch_only_grew_does_not_hide_the_one_before(rt):
    """A graph on stream A uses the scratch, a larger tensor is bound on B, the next graph on C: it waits for A."""
    import time

    import torch

    t, rows, cols, m, wide = T.Q4_K, 2305, 2304, 24, 28928
    rng = np.random.default_rng(7)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    for i in range(2):
        rt.alloc(f"x{i}", m * cols)
        rt.alloc(f"y{i}", m * rows)
        rt.write(f"x{i}", synthetic_activations(m, cols, rng))
        rt.qmv("w", f"x{i}", f"y{i}", m)
    rt.synchronize()
    want = [rt.read_array(f"y{i}", m * rows).copy() for i in range(2)]
    larger = torch.zeros(1024 * wide // 256 * 144 + 256, dtype=torch.uint8, device="cuda")
    graphs = []
    for i in range(2):
        rt.zero(f"y{i}")
        rt.capture_begin()
        rt.qmv("w", f"x{i}", f"y{i}", m)
        graphs.append(rt.capture_end())
    rt.synchronize()
    a, b, c = (torch.cuda.Stream() for _ in range(3))
    done = torch.cuda.Event()
    try:
        with torch.cuda.stream(a):
            torch.cuda._sleep(600_000_000)  # some 0.3 s
        rt.set_stream(a.cuda_stream)
        rt.graph_launch(graphs[0])
        rt.set_stream(b.cuda_stream)
        rt.bind_tensor("larger", larger.data_ptr(), int(t), wide, 1024)
        rt.set_stream(c.cuda_stream)
        rt.graph_launch(graphs[1])
        done.record(c)
        time.sleep(0.05)
        waited = not done.query()
    finally:
        rt.set_stream(None)
        torch.cuda.synchronize()
        for graph in graphs:
            rt.graph_destroy(graph)
    assert waited
    for i in range(2):
        assert np.array_equal(rt.read_array(f"y{i}", m * rows).view(np.uint32), want[i].view(np.uint32)), i
    rt.alloc("xl", m * wide)  # the scratch that grew beside the wait is ready for its first pass
    rt.alloc("yl", m * 1024)
    rt.write("xl", synthetic_activations(m, wide, rng))
    rt.upload("larger", synthetic_blocks(t, 1024, wide, rng), int(t), wide, 1024)
    outs = []
    for run in (lambda work: work(), lambda work: captured(rt, work)):
        run(lambda: rt.qmv("larger", "xl", "yl", m))
        rt.synchronize()
        outs.append(rt.read_array("yl", m * 1024).copy())
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
