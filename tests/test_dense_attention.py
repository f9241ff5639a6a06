"""Dense, rectangular, causal/GQA and fp16 attention through the C ABI against the CPU oracle.

Shapes follow the reference's own primitive tests (tests/pytorch/primitives.py:93-136: odd
lengths 7/128/263, GQA, causal) and its live-mode test (tests/live/attention.py:16-38: the
two-call text/media pattern with row offsets), plus tile-boundary lengths for the 128-row
tcgen05 tiles.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_attention_close

pytestmark = pytest.mark.gpu
SCALE = float(1.0 / np.sqrt(128.0))


def run_sdpa(gpu, oracle, L, H, seed, primitive="sdpa_bf16"):
    q, k, v = (oracle.normal_bf16((1, L, H, 128), seed + i) for i in range(3))
    ty = gpu.empty_bf16(q.size)
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    gpu.call(primitive, ty, tq, tk, tv, L, H, 128, SCALE)
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    want, _ = oracle.attention(q, k, v, SCALE)
    for t in (ty, tq, tk, tv):
        gpu.free(t)
    return got, want


@pytest.mark.parametrize("L", [1, 7, 63, 64, 65, 127, 128, 129, 255, 256, 257, 263, 300, 1000])
def test_sdpa_bf16_lengths(gpu, oracle, L):
    got, want = run_sdpa(gpu, oracle, L, 3, 100 + L)
    assert_attention_close(got, want)
    assert gpu.device_status() == 0


@pytest.mark.parametrize("L,H", [(2048, 8), (1536, 56), (4096, 2)])
def test_sdpa_bf16_larger(gpu, oracle, L, H):
    got, want = run_sdpa(gpu, oracle, L, H, 7 * L + H)
    assert_attention_close(got, want)
    assert gpu.device_status() == 0


@pytest.mark.parametrize("nq,nk,heads", [(64, 9000, 4), (200, 16001, 3), (300, 33000, 2), (1, 5000, 24)])
def test_short_query_block_against_long_keys_split_kv(gpu, oracle, nq, nk, heads):
    """Live mode's text rows against the whole KV history (h3_dit_live.inc:95): too few query tiles
    to fill the GPU, so the keys are cut into slices computed side by side and merged by their
    logsumexp. Same limits as every dense call, ragged last slice included, and the kernel-adapter
    symbol's logsumexp output against the FP32 recomputation."""
    q = oracle.normal_bf16((1, nq, heads, 128), 31)
    k, v = (oracle.normal_bf16((1, nk, heads, 128), 32 + i) for i in range(2))
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    ty = gpu.tensor(np.full(q.shape, 0x7fc0, dtype=np.uint16))
    gpu.call("cross_attention_bf16", ty, 0, tq, 0, tk, tv, 0, nq, nk, heads)
    want, _, want_lse = oracle.attention(q, k, v, SCALE, want_lse=True)
    assert_attention_close(oracle.from_bf16(gpu.read(ty, q.shape)), want)
    tl = gpu.tensor(np.zeros((heads, nq), dtype=np.float32))
    d = gpu.lib.h3b_tensor_data
    gpu.raw("h3_flash3_cross_bf16", d(ty), d(tq), d(tk), d(tv), d(tl), nq, nk, heads, C.c_float(SCALE),
            gpu.lib.h3b_gpu_stream(gpu.gpu))
    assert np.abs(gpu.read(tl, (heads, nq), np.float32) - want_lse.reshape(heads, nq)).max() <= 2e-3
    assert gpu.device_status() == 0


def test_c1_dense_l4096_h8(gpu, oracle):
    """Benchmark configuration 1 exactly: Q, K, V bf16 [1, 8, 4096, 128] from N(0, 1), seed 1001,
    scale 1/sqrt(128), no mask; max-abs <= 1e-2 and cosine >= 0.9999 against the FP32
    recomputation (the whole output, every row)."""
    got, want = run_sdpa(gpu, oracle, 4096, 8, 1001)
    m = assert_attention_close(got, want)
    assert m["rel_l2"] <= 0.004   # the level the reference's own kernel is held to on live shapes
    assert gpu.device_status() == 0


def test_sdpa_fa2_entry_matches_flash3_entry(gpu, oracle):
    """h3_gpu_sdpa_fa2_bf16 (FlashAttention-2 adapter path) and h3_gpu_sdpa_bf16 agree."""
    a, want = run_sdpa(gpu, oracle, 263, 4, 5, "sdpa_bf16")
    b, _ = run_sdpa(gpu, oracle, 263, 4, 5, "sdpa_fa2_bf16")
    assert_attention_close(b, want)
    assert np.array_equal(a, b)


def test_sdpa_uniform_distribution(gpu, oracle):
    """Second input distribution of the reference's attention microbenchmark
    (tests/serving/profile/attn_bench.cu:95-98): Q, K ~ U(-2, 2), V ~ U(-1, 1)."""
    rng = np.random.default_rng(99)
    L, H = 700, 4
    q = oracle.to_bf16(rng.uniform(-2, 2, (1, L, H, 128)))
    k = oracle.to_bf16(rng.uniform(-2, 2, (1, L, H, 128)))
    v = oracle.to_bf16(rng.uniform(-1, 1, (1, L, H, 128)))
    ty = gpu.empty_bf16(q.size)
    gpu.call("sdpa_bf16", ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v), L, H, 128, SCALE)
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    want, _ = oracle.attention(q, k, v, SCALE)
    assert_attention_close(got, want)


def test_sdpa_large_logits_rescale(gpu, oracle):
    """Rows whose maximum keeps growing exercise the lazy accumulator rescale."""
    L, H = 640, 2
    q = oracle.normal_bf16((1, L, H, 128), 41, 3.0)
    k = oracle.from_bf16(oracle.normal_bf16((1, L, H, 128), 42, 1.0))
    k *= np.linspace(0.2, 4.0, L, dtype=np.float32)[None, :, None, None]  # later keys larger
    k = oracle.to_bf16(k)
    v = oracle.normal_bf16((1, L, H, 128), 43)
    ty = gpu.empty_bf16(q.size)
    gpu.call("sdpa_bf16", ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v), L, H, 128, SCALE)
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    want, _ = oracle.attention(q, k, v, SCALE)
    assert_attention_close(got, want, max_abs=2e-2)


@pytest.mark.parametrize("L,H,KH", [(7, 8, 2), (128, 8, 2), (263, 8, 4), (263, 6, 1)])
@pytest.mark.parametrize("causal", [False, True])
def test_flash_bf16_gqa_causal(gpu, oracle, L, H, KH, causal):
    """h3_flash_bf16 directly: causal and grouped-query, batch 2, with logsumexp."""
    B = 2
    q = oracle.normal_bf16((B, L, H, 128), 1000 + L)
    k = oracle.normal_bf16((B, L, KH, 128), 2000 + L)
    v = oracle.normal_bf16((B, L, KH, 128), 3000 + L)
    ty = gpu.empty_bf16(q.size)
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    tl = gpu.tensor(np.zeros((B, H, L), dtype=np.float32))
    data = gpu.lib.h3b_tensor_data
    gpu.raw("h3_flash_bf16", data(ty), data(tq), data(tk), data(tv), data(tl), B, L, H, KH, SCALE,
            causal, gpu.lib.h3b_gpu_stream(gpu.gpu))
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    lse = gpu.read(tl, (B, H, L), np.float32)
    want, _, want_lse = oracle.attention(q, k, v, SCALE, causal=causal, want_lse=True)
    assert_attention_close(got, want)
    assert np.abs(lse - want_lse).max() < 2e-3
    assert gpu.device_status() == 0


def test_gqa_causal_primitive(gpu, oracle):
    """h3_gpu_gqa_causal_bf16 (reference h3_gpu.h:534-540), the text-encoder call."""
    L, H, KH = 150, 16, 2
    q = oracle.normal_bf16((1, L, H, 128), 1)
    k = oracle.normal_bf16((1, L, KH, 128), 2)
    v = oracle.normal_bf16((1, L, KH, 128), 3)
    ty = gpu.empty_bf16(q.size)
    gpu.call("gqa_causal_bf16", ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v), L, H, KH, 128, SCALE)
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    want, _ = oracle.attention(q, k, v, SCALE, causal=True)
    assert_attention_close(got, want)


@pytest.mark.parametrize("L,H", [(7, 2), (64, 3), (263, 4), (1030, 2)])
def test_sdpa_f16_d64(gpu, oracle, L, H):
    """h3_gpu_sdpa_f16_d64: fp16, head dim 64 (video VAE call, reference cuda/vae_fp16.cuh:275-296)."""
    from h3_omni_b200 import native
    rng = np.random.default_rng(L)
    q, k, v = (oracle.to_f16(rng.standard_normal((1, L, H, 64))) for _ in range(3))
    ty = gpu.empty_f16(q.size)
    gpu.call("sdpa_f16_d64", ty, gpu.tensor(q, native.F16), gpu.tensor(k, native.F16),
             gpu.tensor(v, native.F16), L, H, 64, 0.125)
    got = oracle.from_f16(gpu.read(ty, q.shape))
    want, _ = oracle.attention(q, k, v, 0.125, elem="f16")
    assert_attention_close(got, want, max_abs=5e-3, rel_l2=0.004)


@pytest.mark.parametrize("L", [1, 127, 128, 129, 255, 256, 257, 384, 385, 640, 1100])
@pytest.mark.parametrize("shift", [0, 4])
def test_causal_and_f16_at_tile_edges(gpu, oracle, L, shift):
    """The causal and the fp16 head-dim-64 kernels where their tiles end (128-row tiles, two per CTA,
    the diagonal inside or between them), and, with query and output 4 bytes off the 16-byte boundary,
    the kernel that takes such tensors. fp16 limit: half an ulp of values up to 4 plus the rounding of
    the weights (2^-12 each, averaged over the row)."""
    from h3_omni_b200 import native
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
    pad = shift // 2

    def shifted(x, dtype=None):
        return data(gpu.tensor(np.concatenate([np.zeros(pad, np.uint16), x.ravel()]), dtype)) + shift

    B, H, KH = 2, 6, 2
    q = oracle.normal_bf16((B, L, H, 128), 10 + L)
    k, v = (oracle.normal_bf16((B, L, KH, 128), 20 + L + i) for i in range(2))
    ty = gpu.tensor(np.full(q.size + pad, 0x7fc0, dtype=np.uint16))
    tl = gpu.tensor(np.zeros((B, H, L), dtype=np.float32))
    gpu.raw("h3_flash_bf16", data(ty) + shift, shifted(q), data(gpu.tensor(k)), data(gpu.tensor(v)), data(tl), B, L, H,
            KH, SCALE, True, stream)
    want, _, want_lse = oracle.attention(q, k, v, SCALE, causal=True, want_lse=True)
    assert_attention_close(oracle.from_bf16(gpu.read(ty, q.size + pad)[pad:].reshape(q.shape)), want)
    assert np.abs(gpu.read(tl, (B, H, L), np.float32) - want_lse).max() < 2e-3

    rng = np.random.default_rng(L)
    q, k, v = (oracle.to_f16(rng.standard_normal((B, L, 3, 64))) for _ in range(3))
    ty = gpu.tensor(np.full(q.size + pad, 0x7e00, dtype=np.uint16), native.F16)
    gpu.raw("h3_flash3_f16_d64", data(ty) + shift, shifted(q, native.F16), data(gpu.tensor(k, native.F16)),
            data(gpu.tensor(v, native.F16)), None, B, L, 3, 0.125, stream)
    want, _ = oracle.attention(q, k, v, 0.125, elem="f16")
    assert_attention_close(oracle.from_f16(gpu.read(ty, q.size + pad)[pad:].reshape(q.shape)), want, max_abs=2e-3,
                           rel_l2=0.001)
    assert gpu.device_status() == 0


@pytest.mark.parametrize("L", [128, 256, 400, 1100])
def test_causal_and_f16_are_as_exact_as_the_kernel_of_shifted_tensors(gpu, oracle, L):
    """Against 64 bits the tcgen05 kernels are no further off than the mma.sync kernel that takes the same values 4
    bytes off the 16-byte boundary: the output in the 2-norm, and the logsumexp, whose error is that of fp32 scores
    up to about 8 (half an ulp each: 2^-22) and of their fp32 sums of 64 and 128 products."""
    from h3_omni_b200 import native
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)

    def exact(q, k, v, scale, causal):
        s = np.einsum("qhd,khd->hqk", q, np.repeat(k, q.shape[1] // k.shape[1], 1)) * scale
        if causal:
            s[:, np.triu_indices(L, 1)[0], np.triu_indices(L, 1)[1]] = -np.inf
        top = s.max(-1, keepdims=True)
        w = np.exp(s - top)
        out = np.einsum("hqk,khd->qhd", w / w.sum(-1, keepdims=True), np.repeat(v, q.shape[1] // v.shape[1], 1))
        return out, (top + np.log(w.sum(-1, keepdims=True)))[..., 0]

    for f16 in (False, True):
        D, H, KH = (64, 4, 4) if f16 else (128, 6, 2)
        dtype, scale = (native.F16, 0.125) if f16 else (None, SCALE)
        encode, decode = (oracle.to_f16, oracle.from_f16) if f16 else (oracle.to_bf16, oracle.from_bf16)
        rng = np.random.default_rng(L)
        q, k, v = (encode(rng.standard_normal((L, h, D)).astype(np.float32)) for h in (H, KH, KH))
        want, want_lse = exact(*[decode(x).astype(np.float64) for x in (q, k, v)], scale, not f16)
        error = {}
        for pad in (0, 2):
            ty = gpu.tensor(np.zeros(q.size + pad, np.uint16), dtype)
            tq = gpu.tensor(np.concatenate([np.zeros(pad, np.uint16), q.ravel()]), dtype)
            tl = gpu.tensor(np.zeros((H, L), np.float32))
            pointers = [data(ty) + 2 * pad, data(tq) + 2 * pad, *[data(gpu.tensor(x, dtype)) for x in (k, v)], data(tl)]
            if f16:
                gpu.raw("h3_flash3_f16_d64", *pointers, 1, L, H, scale, stream)
            else:
                gpu.raw("h3_flash_bf16", *pointers, 1, L, H, KH, scale, True, stream)
            out = decode(gpu.read(ty, q.size + pad)[pad:].reshape(q.shape))
            error[pad] = np.linalg.norm(out - want)
            assert np.abs(gpu.read(tl, (H, L), np.float32) - want_lse).max() <= 2e-6, (f16, pad)
        assert error[0] <= error[2], (f16, error)


def test_work_memory_is_kept_for_the_next_call_and_given_back(gpu, oracle):
    """The work memory of a call stays with the library when its stream has been waited for, so that the next call
    need not map it again, and goes when a context is freed. Two streams at once get memory of their own."""
    import ctypes as C
    from h3_omni_b200 import native
    rt = native._cudart()

    def free_bytes():
        free, total = C.c_size_t(), C.c_size_t()
        assert rt.cudaDeviceSynchronize() == 0 and rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
        return free.value

    other = native.Native()
    nq, nk, heads = 200, 4500, 8
    q, k, v = (oracle.normal_bf16((n, heads, 128), 90 + n + i) for i, n in enumerate((nq, nk, nk)))
    outs = []
    for _ in range(2):
        for ctx in (gpu, other):
            ty = ctx.empty_bf16(q.size)
            ctx.call("cross_attention_bf16", ty, 0, ctx.tensor(q), 0, ctx.tensor(k), ctx.tensor(v), 0, nq, nk, heads)
            outs.append((ctx, ty))
    got = [ctx.read(ty, q.shape) for ctx, ty in outs]
    assert all(np.array_equal(got[0], x) for x in got[1:])
    for t in list(other.owned):
        other.free(t)
    before = free_bytes()
    other.close()
    assert free_bytes() >= before + (2 << 20)


@pytest.mark.parametrize("column", [0, 2, 66])
def test_not_a_number_in_a_key_reaches_its_rows(gpu, oracle, column):
    """A NaN key makes every row that attends it NaN, whichever unit takes the exponential of its column."""
    from h3_omni_b200 import native
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
    L, key = 400, 128 + column
    q, k, v = (oracle.normal_bf16((1, L, 2, 128), 30 + i) for i in range(3))
    k[0, key, :, 3] = 0x7fc0
    for causal in (False, True):
        ty = gpu.tensor(np.zeros(q.shape, dtype=np.uint16))
        gpu.raw("h3_flash_bf16", *[data(t) for t in (ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v))], None, 1, L, 2, 2,
                SCALE, causal, stream)
        out = oracle.from_bf16(gpu.read(ty, q.shape))[0]
        first = key if causal else 0
        assert np.isnan(out[first:]).all() and np.isfinite(out[:first]).all()
    q, k, v = (oracle.to_f16(np.random.default_rng(40 + i).standard_normal((1, L, 2, 64))) for i in range(3))
    k[0, key, :, 3] = 0x7e00
    ty = gpu.tensor(np.zeros(q.shape, dtype=np.uint16), native.F16)
    gpu.raw("h3_flash3_f16_d64", data(ty), *[data(gpu.tensor(x, native.F16)) for x in (q, k, v)], None, 1, L, 2, 0.125, stream)
    assert np.isnan(oracle.from_f16(gpu.read(ty, q.shape))).all()


@pytest.mark.parametrize("L,first,last", [(256, 130, 131), (384, 256 + 7, 256 + 8), (384, 0, 64), (384, 0, 128), (400, 0, 200),
                                          (400, 300, 400)])
def test_infinite_scores(gpu, oracle, L, first, last):
    """Keys of infinite score: a row of +inf is NaN, whichever unit takes the exponential of which column and also in
    the last tile; a score of -inf is a weight of zero, also when it is all that a row has seen so far (128 keys and
    more in a row; the non-causal bf16 kernel takes fewer)."""
    from h3_omni_b200 import native
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
    for kind in ("dense", "causal", "f16"):
        if kind == "dense" and last - first >= 128:
            continue
        f16 = kind == "f16"
        D, dtype, scale = (64, native.F16, 0.125) if f16 else (128, None, SCALE)
        encode, decode = (oracle.to_f16, oracle.from_f16) if f16 else (oracle.to_bf16, oracle.from_bf16)
        rng = np.random.default_rng(L + last)
        qf, kf, vf = (rng.standard_normal((1, L, 2, D)).astype(np.float32) for _ in range(3))
        qf[..., 3] = np.where(np.abs(qf[..., 3]) < 0.1, 1.0, qf[..., 3])
        q, k, v = encode(qf), encode(kf), encode(vf)
        k[0, first:last, :, 3] = 0x7c00 if f16 else 0x7f80
        ty = gpu.tensor(np.zeros(q.shape, dtype=np.uint16), dtype)
        pointers = [data(ty), *[data(gpu.tensor(x, dtype)) for x in (q, k, v)], None]
        if f16:
            gpu.raw("h3_flash3_f16_d64", *pointers, 1, L, 2, scale, stream)
        else:
            gpu.raw("h3_flash_bf16", *pointers, 1, L, 2, 2, scale, kind == "causal", stream)
        out = decode(gpu.read(ty, q.shape))[0]
        qd, kd, vd = (decode(x)[0].astype(np.float64) for x in (q, k, v))
        kd[first:last, :, 3] = 0.0
        s = np.einsum("qhd,khd->hqk", qd, kd) * scale
        s[:, :, first:last] = -np.inf                       # what a row of negative q[3] sees
        seen = np.tri(L, dtype=bool) if kind == "causal" else np.ones((L, L), dtype=bool)
        s[:, ~seen] = -np.inf
        up = ((qd[..., 3] > 0) & seen[:, first:last].any(1)[:, None]).T
        nothing = np.isneginf(s).all(-1) & ~up
        with np.errstate(invalid="ignore"):
            w = np.exp(s - s.max(-1, keepdims=True))
            want = np.einsum("hqk,khd->hqd", w / w.sum(-1, keepdims=True), vd)
        got = out.transpose(1, 0, 2)
        assert np.isnan(got[up | nothing]).all(), kind
        assert np.abs(got - want)[~(up | nothing)].max() <= 2.5e-2, kind   # few keys: 2^-9 of values up to 4.5, twice
    assert gpu.device_status() == 0


@pytest.mark.parametrize("L,key", [(400, 200), (400, 255), (130, 129), (700, 128), (700, 500), (300, 0)])
def test_causal_rows_see_nothing_of_later_values(gpu, oracle, L, key):
    """An infinite value of a key leaves all rows above the key's group of 64 as they are without it."""
    data, stream = gpu.lib.h3b_tensor_data, gpu.lib.h3b_gpu_stream(gpu.gpu)
    q, k, v = (oracle.normal_bf16((1, L, h, 128), 50 + h) for h in (4, 2, 2))
    got = []
    for value in (None, 0x7f80):
        if value:
            v[0, key, :, 5] = value
        ty = gpu.tensor(np.zeros(q.shape, dtype=np.uint16))
        gpu.raw("h3_flash_bf16", *[data(t) for t in (ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v))], None, 1, L, 4, 2,
                SCALE, True, stream)
        got.append(gpu.read(ty, q.shape)[0])
    above = key // 64 * 64
    assert np.array_equal(got[0][:above], got[1][:above])
    assert not np.isfinite(oracle.from_bf16(got[1])[key:, :, 5]).any()


@pytest.mark.parametrize("kind,L", [("sdpa_bf16", 77), ("sdpa_bf16", 300), ("gqa_causal_bf16", 300), ("sdpa_f16_d64", 300),
                                    ("cross_attention_bf16", 5000)])
def test_calls_that_overlap_see_each_other(gpu, oracle, busy, kind, L):
    """A kernel may be set up while the one before it runs. Calls that read what the call before wrote and write what it
    read (query and output change places), all pending before the first of them starts, give the bits of the same calls
    waited for one by one."""
    from h3_omni_b200 import native
    f16, H = kind == "sdpa_f16_d64", 4
    rows, dtype = (64 if kind == "cross_attention_bf16" else L), native.F16 if f16 else native.BF16
    rng = np.random.default_rng(L)
    make = oracle.to_f16 if f16 else oracle.to_bf16
    q, k, v = (make(rng.standard_normal((n, H, 64 if f16 else 128)).astype(np.float32)) for n in (rows, L, L))
    got = []
    for wait in (True, False):
        a, b, tk, tv = (gpu.tensor(x, dtype) for x in (q, q, k, v))
        if not wait:
            busy.queue()
        for _ in range(12):
            if kind == "cross_attention_bf16":
                gpu.call(kind, b, 0, a, 0, tk, tv, 0, rows, L, H)
            elif kind == "gqa_causal_bf16":
                gpu.call(kind, b, a, tk, tv, L, H, H, 128, SCALE)
            else:
                gpu.call(kind, b, a, tk, tv, L, H, 64 if f16 else 128, SCALE)
            a, b = b, a
            if wait:
                gpu.submit()
        assert wait or busy.running()
        got.append(gpu.read(a, q.shape))
    assert np.array_equal(*got)
    assert gpu.device_status() == 0


def test_sdpa_rejects_bad_arguments(gpu, oracle):
    """Error behaviour of the primitive layer: 0 + message, no launch."""
    q = gpu.tensor(oracle.normal_bf16((4, 2, 128), 1))
    f = gpu.tensor(np.zeros(4 * 2 * 128, dtype=np.float32))
    y = gpu.empty_bf16(4 * 2 * 128)
    with pytest.raises(RuntimeError, match="need 2048 elements"):
        gpu.call("sdpa_bf16", y, q, q, q, 8, 2, 128, SCALE)
    with pytest.raises(RuntimeError, match="expected BF16"):
        gpu.call("sdpa_bf16", y, f, q, q, 4, 2, 128, SCALE)
    with pytest.raises(RuntimeError, match="head dimension 128"):
        gpu.call("sdpa_bf16", y, q, q, q, 4, 4, 64, SCALE)
    assert gpu.lib.h3_flash3_bf16(None, None, None, None, None, 1, 4, 2, 2, SCALE, None) != 0
    assert gpu.lib.h3_flash3_bf16(gpu.lib.h3b_tensor_data(y), gpu.lib.h3b_tensor_data(q),
                                  gpu.lib.h3b_tensor_data(q), gpu.lib.h3b_tensor_data(q), None, 1,
                                  4, 3, 2, SCALE, None) != 0  # 3 heads do not group over 2


def live_case(gpu, oracle, text, media, history, H, seed):
    """Two-call live pattern (reference h3_dit_live.inc:88-99, tests/live/attention.py:16-38):
    K/V rows are [text | history | current media]; text queries attend text only, media
    queries attend everything."""
    total_q = text + media
    total_k = text + history + media
    q = oracle.normal_bf16((total_q, H, 128), seed)
    k = oracle.normal_bf16((total_k, H, 128), seed + 1)
    v = oracle.normal_bf16((total_k, H, 128), seed + 2)
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    ty = gpu.tensor(np.zeros(q.shape, dtype=np.uint16))
    gpu.call("cross_attention_bf16", ty, 0, tq, 0, tk, tv, 0, text, text, H)
    gpu.call("cross_attention_bf16", ty, text, tq, text, tk, tv, 0, media, total_k, H)
    got = oracle.from_bf16(gpu.read(ty, q.shape))
    want_text, _ = oracle.attention(q[None, :text], k[None, :text], v[None, :text], SCALE)
    want_media, _ = oracle.attention(q[None, text:], k[None], v[None], SCALE)
    want = np.concatenate([want_text[0], want_media[0]])
    return got, want


@pytest.mark.parametrize("text,media,history,H", [(17, 100, 0, 4), (77, 300, 500, 4),
                                                   (128, 405, 1215, 7), (5, 64, 3000, 2)])
def test_live_cross_attention(gpu, oracle, text, media, history, H):
    got, want = live_case(gpu, oracle, text, media, history, H, text + media)
    m = assert_attention_close(got, want)
    assert m["rel_l2"] < 0.004  # the reference's own limit, tests/live/attention.py:38
    assert gpu.device_status() == 0


def test_cross_attention_row_offsets_leave_other_rows(gpu, oracle):
    """Output rows outside [out_row, out_row + query_rows) are not touched."""
    H = 2
    q = oracle.normal_bf16((300, H, 128), 5)
    k = oracle.normal_bf16((400, H, 128), 6)
    v = oracle.normal_bf16((400, H, 128), 7)
    sentinel = np.full((300, H, 128), 0x7fc0, dtype=np.uint16)
    ty = gpu.tensor(sentinel)
    gpu.call("cross_attention_bf16", ty, 50, gpu.tensor(q), 20, gpu.tensor(k), gpu.tensor(v), 100,
             130, 250, H)
    out = gpu.read(ty, q.shape)
    assert np.array_equal(out[:50], sentinel[:50]) and np.array_equal(out[180:], sentinel[180:])
    want, _ = oracle.attention(q[None, 20:150], k[None, 100:350], v[None, 100:350], SCALE)
    assert_attention_close(oracle.from_bf16(out[50:180]), want[0])


def test_head_split_is_bit_exact(gpu, oracle):
    """Attention over all heads equals the concatenation of per-half calls bit for bit
    (reference tests/live/sharding.py:38-46): no cross-head arithmetic anywhere."""
    L, H = 333, 8
    q, k, v = (oracle.normal_bf16((L, H, 128), 70 + i) for i in range(3))
    ty = gpu.empty_bf16(q.size)
    gpu.call("sdpa_bf16", ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v), L, H, 128, SCALE)
    full = gpu.read(ty, q.shape)
    halves = []
    for lo in (0, H // 2):
        sl = slice(lo, lo + H // 2)
        th = gpu.empty_bf16(L * (H // 2) * 128)
        gpu.call("sdpa_bf16", th, gpu.tensor(q[:, sl]), gpu.tensor(k[:, sl]), gpu.tensor(v[:, sl]),
                 L, H // 2, 128, SCALE)
        halves.append(gpu.read(th, (L, H // 2, 128)))
    assert np.array_equal(full, np.concatenate(halves, axis=1))


def test_run_twice_is_deterministic(gpu, oracle):
    L, H = 517, 3
    q, k, v = (oracle.normal_bf16((L, H, 128), 80 + i) for i in range(3))
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    outs = []
    for _ in range(2):
        ty = gpu.empty_bf16(q.size)
        gpu.call("sdpa_bf16", ty, tq, tk, tv, L, H, 128, SCALE)
        outs.append(gpu.read(ty, q.shape))
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("groups", [0, 1, 2, 4])
def test_host_buffer_attention_matches_device_path(gpu, oracle, groups):
    """h3b_sdpa_bf16_host (head groups pipelined over copy and compute streams, pageable host
    memory here) gives the same bits as the device-tensor primitive: grouping heads changes
    nothing per head. A second call reuses the staging slots."""
    L, H = 700, 8
    q, k, v = (oracle.normal_bf16((L, H, 128), 90 + i) for i in range(3))
    ty = gpu.empty_bf16(q.size)
    gpu.call("sdpa_bf16", ty, gpu.tensor(q), gpu.tensor(k), gpu.tensor(v), L, H, 128, SCALE)
    want = gpu.read(ty, q.shape)
    for _ in range(2):
        out = np.zeros(q.shape, dtype=np.uint16)
        ok = gpu.lib.h3b_sdpa_bf16_host(gpu.gpu, out.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p),
                                        k.ctypes.data_as(C.c_void_p), v.ctypes.data_as(C.c_void_p), L, H,
                                        128, SCALE, groups)
        assert ok, gpu.error()
        assert np.array_equal(out, want)
    assert not gpu.lib.h3b_sdpa_bf16_host(gpu.gpu, out.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p),
                                          k.ctypes.data_as(C.c_void_p), v.ctypes.data_as(C.c_void_p), L, H,
                                          128, SCALE, 3)
    assert "do not split into 3 groups" in gpu.error()
    assert gpu.device_status() == 0


@pytest.mark.parametrize("nq,ranges,H", [(300, [77, 405, 1000, 128, 300], 4), (64, [5], 2),
                                          (405, [129, 1, 127, 256, 33, 700], 7)])
def test_segmented_live_attention_equals_concatenated(gpu, oracle, nq, ranges, H):
    """h3b_cross_attention_segments_bf16 over separate K/V ranges == h3_gpu_cross_attention_bf16
    over their concatenation (the reference's live path, h3_dit_live.inc:81-99). Ranges that
    are multiples of 128 rows give the same bits; ragged ones regroup the key tiles, so those
    are compared by tolerance and against the oracle."""
    q = oracle.normal_bf16((nq + 9, H, 128), 500)
    ks = [oracle.normal_bf16((r + 3, H, 128), 510 + i) for i, r in enumerate(ranges)]
    vs = [oracle.normal_bf16((r + 3, H, 128), 520 + i) for i, r in enumerate(ranges)]
    kcat = np.concatenate([x[3:] for x in ks])
    vcat = np.concatenate([x[3:] for x in vs])
    tq = gpu.tensor(q)
    want_t = gpu.tensor(np.zeros((nq, H, 128), dtype=np.uint16))
    gpu.call("cross_attention_bf16", want_t, 0, tq, 9, gpu.tensor(kcat), gpu.tensor(vcat), 0, nq, len(kcat), H)
    concat = gpu.read(want_t, (nq, H, 128))
    n = len(ranges)
    tk = (C.c_void_p * n)(*[gpu.tensor(x) for x in ks])
    tv = (C.c_void_p * n)(*[gpu.tensor(x) for x in vs])
    rows = (C.c_uint32 * n)(*ranges)
    offs = (C.c_size_t * n)(*([3] * n))
    out = gpu.tensor(np.zeros((nq + 2, H, 128), dtype=np.uint16))
    ok = gpu.lib.h3b_cross_attention_segments_bf16(gpu.gpu, out, 2, tq, 9, nq, H, n, tk, tv, offs, rows)
    assert ok, gpu.error()
    got = gpu.read(out, (nq + 2, H, 128))
    assert not got[:2].any()
    want, _ = oracle.attention(q[None, 9:], kcat[None], vcat[None], SCALE)
    assert_attention_close(oracle.from_bf16(got[2:]), want[0])
    if all(r % 128 == 0 for r in ranges) or n == 1:
        assert np.array_equal(got[2:], concat)
    else:
        assert np.abs(oracle.from_bf16(got[2:]) - oracle.from_bf16(concat)).max() <= 4e-3
    assert gpu.device_status() == 0
    assert not gpu.lib.h3b_cross_attention_segments_bf16(gpu.gpu, out, 2, tq, 9, nq, H, 7, tk, tv, offs, rows)


@pytest.mark.parametrize("seed", range(12))
def test_random_shapes_against_oracle(gpu, oracle, seed):
    """Seeded random shapes around the tile boundaries of both tcgen05 kernels (128-row query
    tiles, 256-row CTA pairs, 128-row key tiles): a dense call, a rectangular call with row
    offsets, a causal/GQA call and a segmented call per seed, each against the oracle."""
    rng = np.random.default_rng(1000 + seed)
    near = lambda: int(rng.choice([1, 64, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 640]) + rng.integers(0, 3))
    H = int(rng.choice([1, 2, 3, 5]))
    # dense
    L = near()
    got, want = run_sdpa(gpu, oracle, L, H, 3000 + seed)
    assert_attention_close(got, want[0])
    # rectangular with offsets
    nq, nk, qo, ko, oo = near(), near(), int(rng.integers(0, 5)), int(rng.integers(0, 5)), int(rng.integers(0, 5))
    q = oracle.normal_bf16((nq + qo, H, 128), 3100 + seed)
    k = oracle.normal_bf16((nk + ko, H, 128), 3200 + seed)
    v = oracle.normal_bf16((nk + ko, H, 128), 3300 + seed)
    out = gpu.tensor(np.zeros((nq + oo, H, 128), dtype=np.uint16))
    tq, tk, tv = gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    gpu.call("cross_attention_bf16", out, oo, tq, qo, tk, tv, ko, nq, nk, H)
    got = gpu.read(out, (nq + oo, H, 128))
    assert not got[:oo].any()
    want, _ = oracle.attention(q[None, qo:], k[None, ko:], v[None, ko:], SCALE)
    assert_attention_close(oracle.from_bf16(got[oo:]), want[0])
    for t in (out, tq, tk, tv):
        gpu.free(t)
    # causal / grouped-query (the FlashAttention-2 adapter)
    KH = int(rng.choice([1, 2]))
    Hq = KH * int(rng.choice([1, 2, 3]))
    causal = bool(rng.integers(0, 2))
    Lc = near()
    q = oracle.normal_bf16((1, Lc, Hq, 128), 3400 + seed)
    k = oracle.normal_bf16((1, Lc, KH, 128), 3500 + seed)
    v = oracle.normal_bf16((1, Lc, KH, 128), 3600 + seed)
    ty, tq, tk, tv = gpu.empty_bf16(q.size), gpu.tensor(q), gpu.tensor(k), gpu.tensor(v)
    data = gpu.lib.h3b_tensor_data
    gpu.raw("h3_flash_bf16", data(ty), data(tq), data(tk), data(tv), None, 1, Lc, Hq, KH, SCALE, causal,
            gpu.lib.h3b_gpu_stream(gpu.gpu))
    want, _ = oracle.attention(q, k, v, SCALE, causal=causal)
    assert_attention_close(oracle.from_bf16(gpu.read(ty, q.shape)), want)
    for t in (ty, tq, tk, tv):
        gpu.free(t)
    # segmented keys
    n = int(rng.integers(1, 7))
    ranges = [near() for _ in range(n)]
    nq = near()
    q = oracle.normal_bf16((nq, H, 128), 3700 + seed)
    ks = [oracle.normal_bf16((r, H, 128), 3800 + 10 * seed + i) for i, r in enumerate(ranges)]
    vs = [oracle.normal_bf16((r, H, 128), 3900 + 10 * seed + i) for i, r in enumerate(ranges)]
    tensors = [gpu.tensor(x) for x in ks + vs]
    tk = (C.c_void_p * n)(*tensors[:n])
    tv = (C.c_void_p * n)(*tensors[n:])
    rows = (C.c_uint32 * n)(*ranges)
    offs = (C.c_size_t * n)(*([0] * n))
    tq, out = gpu.tensor(q), gpu.tensor(np.zeros((nq, H, 128), dtype=np.uint16))
    assert gpu.lib.h3b_cross_attention_segments_bf16(gpu.gpu, out, 0, tq, 0, nq, H, n, tk, tv, offs, rows), gpu.error()
    want, _ = oracle.attention(q[None], np.concatenate(ks)[None], np.concatenate(vs)[None], SCALE)
    assert_attention_close(oracle.from_bf16(gpu.read(out, (nq, H, 128))), want[0])
    for t in tensors + [tq, out]:
        gpu.free(t)
    assert gpu.device_status() == 0
