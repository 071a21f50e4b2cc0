"""The tensor-core matvec at the sizes where it can go wrong: launches of 72 pieces of 256 x 256 weights and more.

Bars as for the CUDA-core kernel: relative L2 error <= 1e-5 against dequantise + fp64 matvec, a pass of several rows
equal bit for bit to its rows alone, one-hot activations give the dequantised weights.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import dequant_np as O
from vinf_3080ti_b200.gguf_types import F16_FIELDS, TRAITS, GGUFTensorType as T
from vinf_3080ti_b200.synth import synthetic_activations, synthetic_blocks

pytestmark = pytest.mark.gpu
TYPES = [T.Q8_0, T.Q2_K, T.Q3_K, T.Q4_K, T.Q5_K, T.Q6_K, T.IQ2_XXS, T.IQ2_XS, T.IQ3_XXS, T.IQ4_NL, T.IQ3_S, T.IQ2_S, T.IQ4_XS]
REL_L2 = 1e-5


@pytest.fixture(scope="module")
def rt(codebooks):
    from vinf_3080ti_b200.runtime import Runtime

    runtime = Runtime(codebooks["iq3s_grid"], codebooks)
    yield runtime
    runtime.close()


def rel_l2(got, ref) -> float:
    return float(np.linalg.norm(np.asarray(got, dtype=np.float64) - ref) / max(np.linalg.norm(ref), 1e-300))


def _run(rt, names, outs, rows, x):
    rt.alloc("x", x.size)
    rt.write("x", np.ascontiguousarray(x))
    for out, r in zip(outs, rows):
        rt.alloc(out, x.shape[0] * r)
    if len(names) == 1:
        rt.qmv(names[0], "x", outs[0], x.shape[0])
    else:
        rt.qmv_group(names, "x", outs, x.shape[0])
    rt.synchronize()
    return [rt.read_array(out, x.shape[0] * r).reshape(x.shape[0], r).copy() for out, r in zip(outs, rows)]


@pytest.mark.parametrize("shapes,cols", [
    ((9473,), 512),           # 37 tiles and one row, one block per tile, two steps
    ((2305,), 2304),          # columns split over a cluster, an odd number of steps per block
    ((1024, 1000, 24, 8), 2560),  # four tensors, tiles that end inside a tensor, split columns
    ((39000,), 256),          # more tiles than blocks, a single step
], ids=str)
@pytest.mark.parametrize("t", TYPES, ids=lambda t: t.name)
def test_tiles_steps_and_splits_of_every_type(rt, codebooks, t, shapes, cols):
    if t in (T.Q8_0, T.IQ4_NL) and cols > 512:
        cols += 32 * 5  # ends inside a step
    rng = np.random.default_rng(int(t) + sum(shapes) + cols)
    names, outs = [f"w{i}" for i in range(len(shapes))], [f"y{i}" for i in range(len(shapes))]
    raws = [synthetic_blocks(t, rows, cols, rng) for rows in shapes]
    for name, raw, rows in zip(names, raws, shapes):
        rt.upload(name, raw, int(t), cols, rows)
    x = synthetic_activations(8, cols, rng)
    x[1, : cols // 2] *= 1e-6  # a row whose chunks have very different ranges
    x[2] = 0.0
    x[2, [0, cols // 2 + 3, cols - 1][int(t) % 3]] = 1.0  # one-hot
    refs = [O.matvec(raw, int(t), rows, cols, x, codebooks) for raw, rows in zip(raws, shapes)]
    got = _run(rt, names, outs, shapes, x)
    for g, ref in zip(got, refs):
        assert max(rel_l2(g[k], ref[k]) for k in range(8)) <= REL_L2
        if not t.name.endswith(("4_K", "5_K", "2_K")):  # (types with minimums subtract the group's sum in fp32)
            assert np.array_equal(g[2], ref[2].astype(np.float32))
    for m in (1, 2, 3, 5):  # each compiled row count, full and not
        for g, part in zip(got, _run(rt, names, outs, shapes, x[:m])):
            assert np.array_equal(part.view(np.uint32), g[:m].view(np.uint32)), m


@pytest.mark.parametrize("m", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("t", [T.Q3_K, T.Q2_K, T.Q8_0, T.IQ4_NL, T.IQ4_XS], ids=lambda t: t.name)
def test_integer_sums_at_the_ends_of_their_range(rt, codebooks, t, m):
    """Types whose products are summed as integers: the largest and smallest weights times activations whose integers are the largest
    there are, all of one sign, and activations at both ends of fp32's range."""
    rows, cols = 2305, 2304
    block, size = TRAITS[t]
    raw = np.zeros((rows, cols // block, size), dtype=np.uint8)
    raw[1::3] = 0xFF
    raw[2::3] = np.random.default_rng(0).integers(0, 256, raw[2::3].shape, dtype=np.uint8)
    for off in F16_FIELDS[t]:
        raw[:, :, off:off + 2] = np.frombuffer(np.float16(1.0).tobytes(), dtype=np.uint8)
    raw = raw.tobytes()
    x = np.empty((16, cols), dtype=np.float32)
    top = np.float32(2.0) - np.float32(2.0**-23)
    x[0], x[1] = top, -top
    x[2] = np.where(np.arange(cols) % 2, top, -top)
    x[3], x[4] = top * np.float32(2.0**-126), 3 * np.float32(2.0**-149)  # the least normal numbers, subnormal ones
    x[5], x[6] = np.float32(2.0**100), np.float32(2.0**-95)
    x[7] = np.float32(2.0**-97) * np.arange(cols)
    x[8:] = x[:8][::-1]
    bits = 11 if t is T.IQ4_XS else 14  # of the first integer: rounded up to 2^bits with a rest of -1/2, and to an even number with 1/2
    x[8], x[15] = 2.0**bits - 0.5, 1.5 - 2.0**bits
    rt.upload("w", raw, int(t), cols, rows)
    for first in range(0, 16, m):
        (got,) = _run(rt, ["w"], ["y"], (rows,), x[first:first + m])
        ref = O.matvec(raw, int(t), rows, cols, x[first:first + m], codebooks)
        for k in range(m):
            bound = 1e-6 * np.linalg.norm(ref[k]) + 2.0**-149 * np.sqrt(rows)  # fp32 sums over 9 steps; the last place of subnormals
            assert np.linalg.norm(got[k] - ref[k]) <= bound, (first + k, np.linalg.norm(got[k] - ref[k]) / np.linalg.norm(ref[k]))


# The field that a row's first sub-scale (Q8_0: the weight of column 5) is made zero with: (byte, bits kept, bits set)
ZERO_FIRST = {T.Q3_K: [(96, 0xF0, 0), (104, 0xFC, 2)], T.Q2_K: [(0, 0, 0)], T.Q8_0: [(7, 0, 0)], T.IQ4_NL: [(0, 0, 0), (1, 0, 0)],
              T.IQ4_XS: [(4, 0xF0, 0), (2, 0xFC, 2)]}


@pytest.mark.parametrize("m", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("t", list(ZERO_FIRST), ids=lambda t: t.name)
def test_a_row_without_weight_at_an_outlier_is_as_exact_as_without_it(rt, codebooks, t, m):
    """One activation is 10^3 to 10^6 times the others, and every other row's weight there is zero: such a row's error is measured
    against its own products, row by row."""
    rows, cols = 39000, 256
    rng = np.random.default_rng(int(t))
    block, size = TRAITS[t]
    raw = np.frombuffer(synthetic_blocks(t, rows, cols, rng), dtype=np.uint8).reshape(rows, cols // block, size).copy()
    for byte, keep, put in ZERO_FIRST[t]:
        raw[1::2, 0, byte] = raw[1::2, 0, byte] & keep | put

    def weights():
        return O.dequantize(raw.tobytes(), int(t), rows * cols, codebooks).reshape(rows, cols).astype(np.float64)[1::2]

    w, least = weights(), 0.0
    assert not w[:, 5].any()
    rt.upload("w", raw.tobytes(), int(t), cols, rows)
    if t is T.Q2_K:  # a sum over quants and one over minimums, which may cancel
        raw[:, :, 16:80] = 0
        least = weights()
    x = synthetic_activations(16, cols, rng)
    x[:, 5] = 10.0 ** (3 + np.arange(16) % 4) * np.where(np.arange(16) % 8 < 4, 1.0, -1.0)
    rest = x.astype(np.float64)
    rest[:, 5] = 0.0
    for first in range(0, 16, m):
        (got,) = _run(rt, ["w"], ["y"], (rows,), x[first:first + m])
        for k in range(m):
            # fp32: some 40 independent roundings, each of at most 2^-24 of a sum of the order of the products' 2-norm: sqrt(40) of
            # them, and 2.5 times that for the worst of 300000 outputs
            size = np.linalg.norm((w - least) * rest[first + k], axis=1) + np.linalg.norm(least * rest[first + k] + 0 * w, axis=1)
            bound = 2.0**-24 * 16 * size
            error = np.abs(got[k, 1::2] - w @ rest[first + k])
            assert np.all(error <= bound), (first + k, float((error / bound).max()))


@pytest.mark.parametrize("t,rows,cols,ntok", [(T.Q6_K, 9473, 512, 1), (T.Q4_K, 2305, 2304, 4), (T.IQ4_XS, 2305, 2304, 8)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_prologues_residual_and_argmax(rt, codebooks, t, rows, cols, ntok):
    rng = np.random.default_rng(rows + cols + ntok)
    raw = synthetic_blocks(t, rows, cols, rng)
    x, x2 = synthetic_activations(ntok, cols, rng), synthetic_activations(ntok, cols, rng)
    nw = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    rt.upload("w", raw, int(t), cols, rows)
    for name, v in (("x", x), ("x2", x2), ("nw", nw)):
        rt.alloc(name, v.size)
        rt.write(name, v)
    rt.alloc("y", ntok * rows)
    res = rng.standard_normal((ntok, rows)).astype(np.float32)
    rt.write("y", res)
    rt.qmv_fused("w", "x", "y", ntok, add=True, norm="nw", eps=1e-6, silu_mul="x2")
    rt.synchronize()
    ref = O.fused_matvec(raw, int(t), rows, cols, x, codebooks, x2=x2, norm_w=nw, eps=1e-6, residual=res)
    assert rel_l2(rt.read_array("y", ntok * rows).reshape(ntok, rows), ref) <= 2e-5
    ids = rt.qmv_argmax("w", "x", "y", ntok)
    logits = rt.read_array("y", ntok * rows).reshape(ntok, rows)
    assert rel_l2(logits, O.matvec(raw, int(t), rows, cols, x, codebooks)) <= REL_L2
    assert ids == [int(v) for v in logits.argmax(axis=1)]


@pytest.mark.parametrize("ntok", [17, 24, 25, 63])
@pytest.mark.parametrize("t,rows,cols", [(t, 2305, 2304) for t in TYPES] + [(T.Q4_K, 39000, 256), (T.Q6_K, 9473, 512), (T.Q3_K, 1025, 17408)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_twenty_four_rows_at_a_time_equal_eight_bit_for_bit(rt, t, rows, cols, ntok):
    rng = np.random.default_rng(int(t) + rows + ntok)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    x = synthetic_activations(ntok, cols, rng)
    x[1] *= 1e-5
    x[ntok - 1, 7] = np.inf
    (got,) = _run(rt, ["w"], ["y"], (rows,), x)
    for c in range(0, ntok, 8):
        (part,) = _run(rt, ["w"], ["y"], (rows,), x[c:c + 8])
        assert np.array_equal(part.view(np.uint32), got[c:c + 8].view(np.uint32)), c


@pytest.mark.parametrize("ntok", [9, 16, 37])
@pytest.mark.parametrize("t,rows,cols", [(t, 2305, 2304) for t in TYPES] + [(T.Q4_K, 39000, 256), (T.Q6_K, 9473, 512)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_sixteen_rows_at_a_time_equal_eight_bit_for_bit(rt, t, rows, cols, ntok):
    rng = np.random.default_rng(int(t) + rows + ntok)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    x = synthetic_activations(ntok, cols, rng)
    x[1] *= 1e-5
    (got,) = _run(rt, ["w"], ["y"], (rows,), x)
    for c in range(0, ntok, 8):
        (part,) = _run(rt, ["w"], ["y"], (rows,), x[c:c + 8])
        assert np.array_equal(part.view(np.uint32), got[c:c + 8].view(np.uint32)), c


@pytest.mark.parametrize("ntok", [1, 33, 63])
@pytest.mark.parametrize("t,rows,cols", [(T.Q4_K, 257, 512), (T.Q6_K, 70, 2304), (T.Q8_0, 300, 1088), (T.F16, 129, 320)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_prompt_gemm_of_few_rows(rt, codebooks, t, rows, cols, ntok):
    rng = np.random.default_rng(rows + cols + ntok)
    raw = synthetic_blocks(t, rows, cols, rng)
    rt.upload("w", raw, int(t), cols, rows)
    x = synthetic_activations(ntok, cols, rng)
    ref = O.matvec(raw, int(t), rows, cols, x, codebooks)
    rt.set_gemm_min_rows(1)
    try:
        (got,) = _run(rt, ["w"], ["y"], (rows,), x)
    finally:
        rt.set_gemm_min_rows(0)
    assert np.all(np.abs(got - ref) <= 3e-3 * np.abs(ref).max())  # fp16 operands


def _captured_kernels(rt, work) -> list[str]:
    """Names of the kernels that `work` launches when another library (torch) captures the stream."""
    import torch
    from cuda.bindings import driver

    def call(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:] if len(result) > 2 else result[1] if len(result) == 2 else None

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    stream = torch.cuda.Stream()
    try:
        with torch.cuda.graph(graph, stream=stream):
            rt.set_stream(torch.cuda.current_stream().cuda_stream)
            work()
    finally:
        rt.set_stream(None)
    raw = driver.CUgraph(graph.raw_cuda_graph())
    names = []
    for node in call(driver.cuGraphGetNodes(raw, call(driver.cuGraphGetNodes(raw, 0))[1]))[0]:
        if call(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = call(driver.cuGraphKernelNodeGetParams(node))
            name = call(driver.cuKernelGetName(params.kern)) if int(params.kern) else call(driver.cuFuncGetName(params.func))
            names.append(name.decode())
    return names


@pytest.mark.parametrize("extra", [0, 4])  # floats behind 16 rows of x: with some, only the pass shows how many rows there are
def test_the_first_pass_of_sixteen_rows_may_be_captured(codebooks, extra):
    import torch
    from vinf_3080ti_b200.runtime import Runtime

    rng = np.random.default_rng(16)
    shapes = [(T.Q4_K, 2305, 2304), (T.Q6_K, 1025, 17408)]  # the second one wider than the first
    raws = [synthetic_blocks(t, rows, cols, rng) for t, rows, cols in shapes]
    for attempt in range(2):  # (the first runtime of a process loads the kernels, which takes memory)
        runtime = Runtime(codebooks["iq3s_grid"], codebooks)
        try:
            for i, (t, rows, cols) in enumerate(shapes):
                runtime.upload(f"w{i}", raws[i], int(t), cols, rows)
                runtime.alloc(f"x{i}", 16 * cols + extra)
                runtime.alloc(f"y{i}", 16 * rows)
            free = torch.cuda.mem_get_info()[0]
            kernels = _captured_kernels(runtime, lambda: [runtime.qmv(f"w{i}", f"x{i}", f"y{i}", 16) for i in range(2)])
            assert attempt == 0 or extra or torch.cuda.mem_get_info()[0] == free  # allocates nothing
            assert len(kernels) == 4  # per tensor: the B operands, then all 16 rows at once
            assert all("tc_split_kernel" in k or "Li16E" in k for k in kernels), kernels
        finally:
            runtime.close()


def test_the_room_for_wide_passes_is_allocated_once_and_not_for_prompts(codebooks):
    import torch
    from vinf_3080ti_b200.runtime import Runtime

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    shapes = [(T.Q4_K, 2305, 2304), (T.Q4_K, 1025, 17408), (T.Q6_K, 1025, 24576)]
    weights = [torch.zeros(rows * (cols // 256) * TRAITS[t][1] + 256, dtype=torch.uint8, device="cuda") for t, rows, cols in shapes]
    x = torch.zeros(512 * 2304, device="cuda")
    runtime = Runtime(codebooks["iq3s_grid"], codebooks)
    try:
        runtime.bind_tensor("w0", weights[0].data_ptr(), int(T.Q4_K), 2304, 2305)
        before = free()
        runtime.bind("prompt", x.data_ptr(), 512 * 2304)
        runtime.set_gemm_min_rows(64)
        runtime.bind("more", x.data_ptr(), 64 * 2304)
        assert free() == before
        runtime.bind("x", x.data_ptr(), 24 * 2304)
        made = free()
        assert made < before
        for i, (t, rows, cols) in enumerate(shapes):
            runtime.bind_tensor(f"w{i}", weights[i].data_ptr(), int(t), cols, rows)
        runtime.set_gemm_min_rows(0)
        assert free() == made
    finally:
        runtime.close()


@pytest.mark.parametrize("t", TYPES, ids=lambda t: t.name)
def test_infinite_and_undefined_activations(rt, codebooks, t):
    """An output is infinite or undefined exactly where weight times activation makes it so, as on the CUDA cores; the other
    activation rows of the pass do not notice."""
    rng = np.random.default_rng(int(t))
    rows, cols = 2305, 2304
    raw = synthetic_blocks(t, rows, cols, rng)
    w = O.dequantize(raw, int(t), rows * cols, codebooks).reshape(rows, cols).astype(np.float64)
    x = synthetic_activations(12, cols, rng)
    x[0, 700] = np.inf
    x[1, [3, 2303]] = np.inf, -np.inf
    x[2, 1111] = np.nan
    x[3, 600] = -np.inf
    with np.errstate(invalid="ignore"):
        want = x[:4].astype(np.float64)[:, None, :] * w[None]
        want = want.sum(axis=2)
    rt.upload("w", raw, int(t), cols, rows)
    (plain,) = _run(rt, ["w"], ["y"], (rows,), np.where(np.isfinite(x), x, np.float32(0)))
    for m in (12, 8, 4, 1):
        (got,) = _run(rt, ["w"], ["y"], (rows,), x[:m])
        for k in range(min(m, 4)):
            assert np.array_equal(np.isnan(got[k]), np.isnan(want[k])) and not np.isfinite(got[k]).any(), (m, k)
            assert np.array_equal(np.sign(got[k][~np.isnan(got[k])]), np.sign(want[k][~np.isnan(want[k])])), (m, k)
        assert np.array_equal(got[4:].view(np.uint32), plain[4:m].view(np.uint32)), m
    nw, x2 = rng.uniform(0.5, 1.5, cols).astype(np.float32), synthetic_activations(4, cols, rng)
    for name, v in (("x", x[:4]), ("x2", x2), ("nw", nw)):
        rt.alloc(name, v.size)
        rt.write(name, np.ascontiguousarray(v))
    rt.alloc("y", 4 * rows)
    outs = []
    for split in (True, False):  # the tensor cores and the CUDA cores
        rt.set_column_split(split)
        try:
            for fuse in ({"silu_mul": "x2"}, {"norm": "nw"}):
                rt.qmv_fused("w", "x", "y", 4, **fuse)
                rt.synchronize()
                outs.append(rt.read_array("y", 4 * rows).copy())
        finally:
            rt.set_column_split(True)
    for a, b in zip(outs[:2], outs[2:]):
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))


@pytest.mark.parametrize("what", ["tall", "tall argmax", "24 rows", "short", "prompt"])
def test_launch_count_is_the_number_of_kernels(rt, what):
    import torch

    t, rows, cols, m = T.Q4_K, 2305, 2304, 4
    if "tall" in what:  # one tile more than SMs: the last one's columns are split, in a launch of its own
        rows, cols = 256 * torch.cuda.get_device_properties(0).multi_processor_count + 256, 2560
    elif what == "24 rows":
        m = 24
    elif what == "short":
        rows = 48
    rt.upload("w", synthetic_blocks(t, rows, cols, np.random.default_rng(3)), int(t), cols, rows)
    rt.alloc("x", m * cols)
    rt.alloc("y", m * rows)
    if what == "tall argmax":
        work = lambda: rt.qmv_argmax("w", "x", "y", m, blocking=False)  # noqa: E731
    else:
        work = lambda: rt.qmv("w", "x", "y", m)  # noqa: E731
    if what == "prompt":
        rt.set_gemm_min_rows(1)
    try:
        work()
        rt.synchronize()
        before = rt.launch_count()
        kernels = _captured_kernels(rt, work)
    finally:
        rt.set_gemm_min_rows(0)
    assert rt.launch_count() - before == len(kernels) == {"24 rows": 3, "short": 1}.get(what, 2)


@pytest.mark.parametrize("graph", [False, True])
def test_wide_passes_on_two_streams_take_turns(rt, graph):
    """The B operands of a pass of more than 8 rows lie in scratch of the runtime: on another stream the next such pass waits."""
    import time

    import torch

    t, rows, cols, m = T.Q4_K, 2305, 2304, 24
    rng = np.random.default_rng(24)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    xs = [synthetic_activations(m, cols, rng) for _ in range(2)]
    for i in range(2):
        rt.alloc(f"x{i}", m * cols)
        rt.alloc(f"y{i}", m * rows)
        rt.write(f"x{i}", xs[i])
        rt.qmv("w", f"x{i}", f"y{i}", m)
    rt.synchronize()
    want = [rt.read_array(f"y{i}", m * rows).copy() for i in range(2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ids = []
    for i in range(2):
        rt.zero(f"y{i}")
        rt.capture_begin()
        rt.qmv("w", f"x{i}", f"y{i}", m)
        ids.append(rt.capture_end())
    rt.synchronize()
    done = torch.cuda.Event()
    try:
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(600_000_000)  # some 0.3 s
        for i in range(2):
            rt.set_stream(streams[i].cuda_stream)
            if graph:
                rt.graph_launch(ids[i])
            else:
                rt.qmv("w", f"x{i}", f"y{i}", m)
        done.record(streams[1])
        time.sleep(0.05)
        waited = not done.query()
    finally:
        rt.set_stream(None)
        torch.cuda.synchronize()
        for g in ids:
            rt.graph_destroy(g)
    assert waited
    for i in range(2):
        assert np.array_equal(rt.read_array(f"y{i}", m * rows).view(np.uint32), want[i].view(np.uint32)), i


def _captured(rt, work):
    """`work` as a graph, launched once: in a capture the blocks that share columns are clusters."""
    rt.capture_begin()
    work()
    graph = rt.capture_end()
    rt.graph_launch(graph)
    rt.synchronize()
    rt.graph_destroy(graph)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 7, 8, 9, 16, 17, 24])
@pytest.mark.parametrize("t", [T.Q6_K, T.Q3_K, T.Q8_0, T.IQ3_S], ids=lambda t: t.name)
@pytest.mark.parametrize("rows,cols", [(2305, 2304), (1030, 5120), (4099, 1280)], ids=str)
def test_sums_exchanged_through_memory_and_in_clusters_are_the_same(rt, t, rows, cols, m):
    rng = np.random.default_rng(rows + cols + m)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    rt.alloc("x", m * cols)
    rt.alloc("y", m * rows)
    for _ in range(2):  # the second launch finds what the first has left behind
        rt.write("x", synthetic_activations(m, cols, rng))
        outs = []
        for run in (lambda work: work(), lambda work: _captured(rt, work)):
            rt.zero("y")
            run(lambda: rt.qmv("w", "x", "y", m))
            rt.synchronize()
            outs.append(rt.read_array("y", m * rows).copy())
        assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
        assert np.abs(outs[0]).max() > 0


@pytest.mark.parametrize("m", [1, 2, 4, 5, 8])
def test_fused_sums_exchanged_through_memory_and_in_clusters_are_the_same(rt, m):
    t, rows, cols = T.Q6_K, 2305, 2304
    rng = np.random.default_rng(m)
    rt.upload("w", synthetic_blocks(t, rows, cols, rng), int(t), cols, rows)
    for name, n in (("x", m * cols), ("x2", m * cols), ("g", cols), ("y0", m * rows), ("y", m * rows)):
        rt.alloc(name, n)
    for name, n in (("x", m), ("x2", m), ("g", 1)):
        rt.write(name, synthetic_activations(n, cols, rng))
    rt.write("y0", synthetic_activations(m, rows, rng))
    for options in ({"norm": "g"}, {"norm": "g", "add": True}, {"silu_mul": "x2", "add": True}):
        outs = []
        for run in (lambda work: work(), lambda work: _captured(rt, work)):
            rt.copy("y", 0, "y0", 0, m * rows)
            run(lambda: rt.qmv_fused("w", "x", "y", m, **options))
            rt.synchronize()
            outs.append(rt.read_array("y", m * rows).copy())
        assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32)), options
    ids = []
    for run in (lambda work: work(), lambda work: _captured(rt, work)):
        run(lambda: rt.qmv_argmax("w", "x", "y", m, blocking=False))
        ids.append(rt.argmax_fetch(m))
    assert ids[0] == ids[1] == rt.read_array("y", m * rows).reshape(m, rows).argmax(axis=1).tolist()


def test_overlapping_streams_and_more_runtimes_than_rooms_for_sums(codebooks):
    import torch
    from vinf_3080ti_b200.runtime import Runtime

    t, rows, cols, m = T.Q4_K, 2305, 2304, 4
    rng = np.random.default_rng(3)
    raw, xs = synthetic_blocks(t, rows, cols, rng), [synthetic_activations(m, cols, rng) for _ in range(3)]
    runtimes = [Runtime(codebooks["iq3s_grid"], codebooks) for _ in range(18)]
    try:
        want = None
        for rt in runtimes:
            rt.upload("w", raw, int(t), cols, rows)
            for i, x in enumerate(xs):
                rt.alloc(f"x{i}", m * cols)
                rt.alloc(f"y{i}", m * rows)
                rt.write(f"x{i}", x)
        for rt in runtimes:
            streams = [None] + [torch.cuda.Stream() for _ in range(5)]
            for k in range(12):  # one runtime, launches on six streams that wait for nothing
                stream = streams[k % 6]
                rt.set_stream(stream.cuda_stream if stream is not None else None)
                if k >= 3 and stream is not None:
                    stream.synchronize()
                rt.qmv("w", f"x{k % 3}", f"y{k % 3}", m)
            torch.cuda.synchronize()
            rt.set_stream(None)
            rt.synchronize()
            got = [rt.read_array(f"y{i}", m * rows).copy() for i in range(3)]
            want = want or got
            for g, w in zip(got, want):
                assert np.array_equal(g.view(np.uint32), w.view(np.uint32))
        ref = O.matvec(raw, int(t), rows, cols, xs[0], codebooks)
        assert rel_l2(want[0].reshape(m, rows), ref) <= REL_L2
    finally:
        for rt in runtimes:
            rt.close()
