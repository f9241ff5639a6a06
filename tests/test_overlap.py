"""Kernels that are set up while the one before them in the stream still runs: what they may read and when, and rows of
different calls that depend on each other without a wait in between."""
import ctypes as C
import re

import numpy as np
import pytest

from conftest import ROOT, ROPE_HALF, out_proj_inputs, rope_inputs

SCALE = float(1 / np.sqrt(128))
CSRC = ROOT / "h3-omni_b200" / "csrc"
OVERLAPPED = sorted(p.name for p in CSRC.glob("*.cu") if "launch_overlapped(" in p.read_text())


def code_of(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


@pytest.mark.parametrize("name", OVERLAPPED + ["softmax_tc5.cuh", "sm100_ptx.cuh", "sparse_choice.cuh"])
def test_overlapped_kernels_read_by_ordinary_loads(name):
    """Their inputs may be written while they are resident: no read-only path, asked for or left to the compiler."""
    assert not re.findall(r"__ldg\b|__restrict__|\.nc\b", code_of(CSRC / name))


@pytest.mark.parametrize("name", OVERLAPPED)
def test_overlapped_kernels_wait_before_they_allow_the_next(name):
    code = code_of(CSRC / name)
    starts = [m.start() for m in re.finditer(r"__global__", code)]
    assert starts
    for begin, end in zip(starts, starts[1:] + [len(code)]):
        body = code[begin:end]
        assert "wait_for_previous_kernel()" in body
        assert body.index("wait_for_previous_kernel()") < body.index("allow_next_kernel()")


@pytest.mark.gpu
@pytest.mark.parametrize("heads,shape", [(3, (7, 8, 8)), (8, (37, 15, 27)), (7, (20, 30, 54))])
def test_static_topk_in_a_row_with_changing_inputs(gpu, oracle, busy, heads, shape):
    """Pooling and selection alternate with nothing between, and every call overwrites the pooled means the selection
    before it read: the lists of each call are those of the call made alone."""
    handle = gpu.call("vsa_new", 17, 30, *shape, heads)
    try:
        info = [C.c_int() for _ in range(4)]
        assert gpu.lib.h3b_vsa_info(handle, *[C.byref(x) for x in info])
        rows, tiles, prefix, keep = (x.value for x in info)
        data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
        tables = [gpu.lib.h3b_vsa_buffer(handle, which) for which in (0, 1)]
        inputs = [[gpu.tensor(oracle.normal_bf16((rows, heads, 128), 61 + 2 * i + j)) for j in range(2)] for i in range(3)]
        got = []
        for wait in (True, False):
            lists = [[gpu.tensor(np.full(s, -7, dtype=np.int32)) for s in ((heads, tiles, tiles), (heads, tiles))]
                     for _ in range(6)]
            if not wait:
                busy.queue()
            for n, (indices, counts) in enumerate(lists):
                q, k = inputs[n % 3]
                assert gpu.lib.h3b_vsa_topk_static(data(q), data(k), *tables, data(indices), data(counts), tiles, prefix,
                                                   keep, heads, stream) == 0
                if wait:
                    gpu.submit()
            assert wait or busy.running()
            got.append([gpu.read(t, s, np.int32) for pair in lists
                        for t, s in zip(pair, ((heads, tiles, tiles), (heads, tiles)))])
        assert not np.array_equal(got[0][0], got[0][2])
        assert all(np.array_equal(a, b) for a, b in zip(*got))
        assert gpu.device_status() == 0
    finally:
        gpu.lib.h3_gpu_vsa_free(handle)


def both_ways(gpu, busy, make, step, steps, result, others=()):
    """The results of `steps` calls of step(state, n) waited for one by one, and of the same calls all pending before the
    first of them starts."""
    got = []
    for wait in (True, False):
        state = make()
        if not wait:
            busy.queue()
        for n in range(steps):
            step(state, n)
            if wait:
                for context in (gpu, *others):
                    context.submit()
        assert wait or busy.running()
        got.append(result(state))
    assert gpu.device_status() == 0
    return got


class Block:
    """Norm + RoPE, dense attention, output projection + gate + AdaLN, over one set of buffers. The projection is as wide as
    Q, K and V together, so that the AdaLN rows are the next step's input; gate and residual accumulate in place."""

    def __init__(self, gpu, oracle, rows, heads):
        self.gpu, self.rows, self.heads, self.hidden = gpu, rows, heads, 3 * heads * 128
        x, w, residual, norm, modulation, row_map = out_proj_inputs(oracle, rows, heads * 128, self.hidden, 40 + rows)
        self.tables = [gpu.tensor(t) for t in rope_inputs(oracle, rows, heads, 41)]
        self.weights = [gpu.tensor(t) for t in (w, norm, modulation, row_map)]
        self.residual, self.row = gpu.tensor(residual), self.tables.pop(0)
        self.q, self.k, self.v, self.attended = (gpu.empty_bf16(rows * heads * 128) for _ in range(4))

    def step(self):
        gpu, (w, norm, modulation, row_map) = self.gpu, self.weights
        gpu.call("grouped_qkv_rope_bf16", self.q, self.k, self.v, self.row, *self.tables, self.rows, self.heads, 128, ROPE_HALF, 1e-5)
        gpu.call("sdpa_bf16", self.attended, self.q, self.k, self.v, self.rows, self.heads, 128, SCALE)
        assert gpu.lib.h3b_attention_output_gate_adaln_bf16(
            gpu.gpu, self.residual, self.row, self.residual, self.attended, w, norm, modulation, modulation, row_map, self.rows,
            self.heads * 128, self.hidden, 6, 2, 3, 4, C.c_float(1e-5)), gpu.error()

    def result(self):
        read = self.gpu.read
        return [read(t, (self.rows, self.hidden)) for t in (self.residual, self.row)] + \
            [read(t, (self.rows, self.heads * 128)) for t in (self.q, self.k, self.v, self.attended)]


@pytest.mark.gpu
@pytest.mark.parametrize("rows,heads", [(77, 2), (300, 4), (1300, 3)])
def test_blocks_in_a_row(gpu, oracle, busy, rows, heads):
    a, b = both_ways(gpu, busy, lambda: Block(gpu, oracle, rows, heads), lambda s, n: s.step(), 6, Block.result)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,heads", [((7, 8, 8), 3), ((12, 15, 27), 6)])
def test_fused_sparse_calls_in_a_row(gpu, oracle, busy, shape, heads):
    """One object, another projection output every time, and each call's output is the gate of the next."""
    handle = gpu.call("vsa_new", 17, 30, *shape, heads)
    try:
        rows = 47 + int(np.prod(shape))
        inputs = [[gpu.tensor(t) for t in rope_inputs(oracle, rows, heads, 90 + i)] for i in range(3)]
        gate = oracle.normal_bf16((rows, heads, 128), 95, 0.3)

        def step(tensors, n):
            assert gpu.lib.h3b_vsa_qkv_rope_bf16(handle, tensors[n + 1], *inputs[n % 3], tensors[n], ROPE_HALF,
                                                 C.c_float(1e-5), 1), gpu.error()

        a, b = both_ways(gpu, busy, lambda: [gpu.tensor(gate)] + [gpu.empty_bf16(gate.size) for _ in range(6)], step, 6,
                         lambda tensors: [gpu.read(t, gate.shape) for t in tensors])
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    finally:
        gpu.lib.h3_gpu_vsa_free(handle)


@pytest.mark.gpu
def test_calls_with_several_key_ranges_in_a_row(gpu, oracle, busy):
    """Query, keys, values and output are three tensors that change places: every call reads what the two before it wrote."""
    rows, heads, ranges = 260, 3, (260, 33)
    first = [oracle.normal_bf16((rows, heads, 128), 100 + i) for i in range(3)]

    def step(t, n):
        x, y, out = (t[(n + i) % 3] for i in range(3))
        assert gpu.lib.h3b_cross_attention_segments_bf16(
            gpu.gpu, out, 0, x, 0, rows, heads, 2, (C.c_void_p * 2)(x, y), (C.c_void_p * 2)(y, x), (C.c_size_t * 2)(0, 7),
            (C.c_uint32 * 2)(*ranges)), gpu.error()

    a, b = both_ways(gpu, busy, lambda: [gpu.tensor(x) for x in first], step, 9,
                     lambda t: [gpu.read(x, first[0].shape) for x in t])
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
def test_two_streams_at_once(gpu, oracle, busy):
    """Waiting kernels hold tensor memory while kernels of another stream come and go: both rows end, with the bits each
    has alone."""
    from h3_omni_b200 import native
    other = native.Native()
    handle = other.call("vsa_new", 17, 30, 7, 8, 8, 3)
    try:
        rows = 47 + 7 * 8 * 8
        sparse = [oracle.normal_bf16((rows, 3, 128), 110 + i) for i in range(4)]

        def make():
            return Block(gpu, oracle, 300, 4), [other.tensor(x) for x in sparse] + [other.empty_bf16(sparse[0].size)]

        def step(state, n):
            block, (q, k, v, gate, out) = state
            block.step()
            src, dst = (q, out) if n % 2 == 0 else (out, q)
            assert other.lib.h3_gpu_vsa_bf16(handle, dst, src, k, v, gate), other.error()
            other.call("sdpa_bf16", src, dst, k, v, rows, 3, 128, SCALE)

        a, b = both_ways(gpu, busy, make, step, 12,
                         lambda s: s[0].result() + [other.read(t, sparse[0].shape) for t in s[1]], (other,))
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    finally:
        other.lib.h3_gpu_vsa_free(handle)
        other.close()


@pytest.mark.gpu
def test_a_captured_row_of_calls(gpu, oracle):
    """Dense, split-key, sparse and projection calls captured in one graph and replayed, against the same calls made directly."""
    from h3_omni_b200 import native
    runtime, stream = native._cudart(), C.c_void_p(gpu.lib.h3b_gpu_stream(gpu.gpu))
    handle = gpu.call("vsa_new", 17, 30, 7, 8, 8, 4)
    graph, executable = C.c_void_p(), C.c_void_p()
    try:
        rows, heads = 47 + 7 * 8 * 8, 4
        gate, keys = oracle.normal_bf16((rows, heads, 128), 120, 0.3), oracle.normal_bf16((5000, heads, 128), 121)

        def make():
            return Block(gpu, oracle, rows, heads), gpu.tensor(gate), gpu.tensor(keys), gpu.empty_bf16(gate.size)

        def step(state):
            block, tg, tk, out = state
            block.step()
            assert gpu.lib.h3_gpu_vsa_bf16(handle, out, block.attended, block.k, block.v, tg), gpu.error()
            gpu.call("cross_attention_bf16", tg, 0, out, 0, tk, tk, 0, 64, 5000, heads)   # (its first 64 rows)

        def result(state):
            return state[0].result() + [gpu.read(t, gate.shape) for t in (state[1], state[3])]

        direct, replayed = make(), make()
        for _ in range(3):
            step(direct)
            gpu.submit()
        assert runtime.cudaStreamBeginCapture(stream, 1) == 0   # thread-local
        step(replayed)
        assert runtime.cudaStreamEndCapture(stream, C.byref(graph)) == 0
        assert runtime.cudaGraphInstantiate(C.byref(executable), graph, C.c_ulonglong(0)) == 0
        for _ in range(3):
            assert runtime.cudaGraphLaunch(executable, stream) == 0
        gpu.submit()
        assert all(np.array_equal(x, y) for x, y in zip(result(direct), result(replayed)))
        assert gpu.device_status() == 0
    finally:
        if executable:
            runtime.cudaGraphExecDestroy(executable)
        if graph:
            runtime.cudaGraphDestroy(graph)
        gpu.lib.h3_gpu_vsa_free(handle)


@pytest.mark.gpu
def test_a_refused_launch_leaves_no_error_behind(gpu, oracle):
    """A grid of more heads than the launch takes is refused by the runtime. The code comes back from that call, and the
    next one, a kernel launched and checked in the ordinary way (an output off 16-byte boundaries), succeeds."""
    heads, L = 65536, 20
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
    pooled = gpu.tensor(np.zeros((heads, 1, 128), dtype=np.float32))
    lists = [gpu.tensor(np.full(heads, -7, dtype=np.int32)) for _ in range(2)]
    q, k, v = (gpu.tensor(oracle.normal_bf16((L, 1, 128), 71 + i)) for i in range(3))
    want, out = gpu.tensor(np.zeros((L, 128), dtype=np.uint16)), gpu.tensor(np.zeros((L + 1, 128), dtype=np.uint16))
    assert gpu.lib.h3b_vsa_select_raw(data(pooled), data(pooled), None, None, data(lists[0]), data(lists[1]), None, 1, 0, 1,
                                      heads, stream) != 0
    gpu.raw("h3_flash_bf16", data(out) + 4, data(q), data(k), data(v), None, 1, L, 1, 1, 0.0883883476, True, stream)
    gpu.raw("h3_flash_bf16", data(want), data(q), data(k), data(v), None, 1, L, 1, 1, 0.0883883476, True, stream)
    got = gpu.read(out, ((L + 1) * 128,))[2:2 + L * 128]
    # Values below 4: either result is within half a bf16 step (2^-7) and its weights' rounding (2^-9 of 4) of the exact one.
    got, want = oracle.from_bf16(got), oracle.from_bf16(gpu.read(want, (L * 128,)))
    assert np.abs(want).max() < 4 and np.abs(got - want).max() <= 2.0 ** -5
    assert all(np.array_equal(gpu.read(t, (heads,), np.int32), np.full(heads, -7, dtype=np.int32)) for t in lists)
