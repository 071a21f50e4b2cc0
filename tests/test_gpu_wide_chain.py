"""Passes of 9 to 24 rows that follow one another on a stream: the kernel that makes the B operands reads what the pass before has left."""
from __future__ import annotations

import numpy as np
import pytest

from vinf_3080ti_b200.gguf_types import GGUFTensorType as T
from vinf_3080ti_b200.synth import synthetic_activations, synthetic_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [9, 16, 17, 24])
@pytest.mark.parametrize("t", [T.Q6_K, T.Q3_K], ids=lambda t: t.name)
def test_passes_that_feed_one_another_are_the_same_with_and_without_waiting(codebooks, t, m):
    from vinf_3080ti_b200.runtime import Runtime

    n, passes = 2304, 12
    rng = np.random.default_rng(m)
    rt = Runtime(codebooks["iq3s_grid"], codebooks)
    try:
        rt.upload("w", synthetic_blocks(t, n, n, rng), int(t), n, n)
        rt.alloc("t", m * n)
        for i in range(passes):
            rt.alloc(f"x{i}", m * n)
            rt.alloc(f"y{i}", m * n)
            rt.write(f"x{i}", synthetic_activations(m, n, rng))
        outs = []
        for wait in (True, False):
            for i in range(passes):
                rt.zero(f"y{i}")
            rt.zero("t")
            rt.synchronize()
            for i in range(passes):  # "t" is both pass's output and the next one's input, for all of them
                for src, dst in ((f"x{i}", "t"), ("t", f"y{i}")):
                    rt.qmv("w", src, dst, m)
                    if wait:
                        rt.synchronize()
            rt.synchronize()
            outs.append([rt.read_array(f"y{i}", m * n).copy() for i in range(passes)])
        for i, (a, b) in enumerate(zip(*outs)):
            assert np.isfinite(a).all() and np.abs(a).max() > 0
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), i
    finally:
        rt.close()
