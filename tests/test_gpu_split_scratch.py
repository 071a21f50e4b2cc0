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
