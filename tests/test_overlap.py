"""Kernels that are set up while the one before them in the stream still runs: what they may read and when, and rows of
different calls that depend on each other without a wait in between."""
import ctypes as C
import re

import numpy as np
import pytest

from conftest import ROOT

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


class Busy:
    """An ordinary call of about two milliseconds: what is queued behind it is pending before any of it starts."""

    def __init__(self, gpu):
        self.gpu, self.rows, self.heads = gpu, 14000, 24
        zero = np.zeros((self.rows, self.heads, 128), dtype=np.uint16)
        self.out, self.x = gpu.tensor(zero), gpu.tensor(zero)

    def queue(self):
        self.gpu.call("sdpa_bf16", self.out, self.x, self.x, self.x, self.rows, self.heads, 128, 0.0883883476)

    def close(self):
        for t in (self.out, self.x):
            self.gpu.free(t)


@pytest.fixture(scope="module")
def busy(gpu):
    b = Busy(gpu)
    yield b
    b.close()


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
            got.append([gpu.read(t, s, np.int32) for pair in lists
                        for t, s in zip(pair, ((heads, tiles, tiles), (heads, tiles)))])
        assert not np.array_equal(got[0][0], got[0][2])
        assert all(np.array_equal(a, b) for a, b in zip(*got))
        assert gpu.device_status() == 0
    finally:
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
