"""The attention work this library is used for, as calls through its C ABI.

listed() names the representative calls of a diffusion transformer's block (and of the text
encoder and video decoder beside it), draw() gives further sizes of the same ranges, prepare() makes
what a caller holds before the call, run() makes the call, work() counts what it cannot do without
and tolerance() says how far two correct implementations may differ.
"""
import ctypes as C
import math

import torch

from __graft_entry__ import load_package

load_package()
from h3_omni_b200 import native  # noqa: E402

DIM = 128
SCALE = 1.0 / math.sqrt(DIM)
ROPE_HALF = 48
EPSILON = 1e-5
HIDDEN = 5376          # width of the residual stream
SLOTS = 6              # modulation vectors per row group
LARGEST_FLOPS = 34e12  # what the largest listed call does; a drawn call does no more
ADD_BYTES = 2          # bytes of a bf16 or fp16 value


def listed():
    return [
        # A text refiner layer: a prompt's tokens among themselves. One small kernel; latency counts.
        {"name": "text_refiner", "kind": "refine", "rows": 77, "heads": 24},
        # A text encoder layer: causal, grouped-query, a long prompt of no round length.
        {"name": "text_encoder", "kind": "causal", "rows": 1000, "heads": 32, "kv_heads": 8},
        # A video decoder attention layer: fp16, head dim 64, one 64 x 64 latent tile.
        {"name": "video_decoder", "kind": "decode", "rows": 4096, "heads": 8},
        # Norm + RoPE before dense attention, five seconds of 864x480 (37 frames of 15x27 tokens + text and audio).
        {"name": "norm_rope_5s", "kind": "rope", "rows": 15400, "heads": 56, "grouped": True},
        # Dense joint attention of that clip: the call every block of the original mode makes.
        {"name": "dense_5s", "kind": "dense", "rows": 15400, "heads": 56, "sharp": 2.0},
        # The long benchmark sequence (51,840 video + 512 audio tokens).
        {"name": "dense_long", "kind": "dense", "rows": 52352, "heads": 24, "sharp": 1.0},
        # The same call from and to pinned host memory, as a program without device tensors makes it.
        {"name": "dense_5s_host", "kind": "host", "rows": 15400, "heads": 56},
        # Output projection + gate + residual + AdaLN after that attention.
        {"name": "projection_5s", "kind": "project", "rows": 15400, "heads": 56},
        # Fast mode: video sparse attention of the five second clip, neighbouring tokens alike.
        {"name": "sparse_5s", "kind": "sparse", "text": 100, "audio": 315, "time": 37, "height": 15, "width": 27,
         "heads": 56, "alike": True, "fused": False, "kept": 0.1},
        # Fast mode at the long benchmark size, fed by the projection output, independent tokens.
        {"name": "sparse_long", "kind": "sparse", "text": 64, "audio": 512, "time": 32, "height": 30, "width": 54,
         "heads": 24, "alike": False, "fused": True, "kept": 0.125},
        # Live mode: the text rows of a block against the whole key history.
        {"name": "live_text", "kind": "live_text", "rows": 256, "keys": 64800, "heads": 24},
        # Live mode: a chunk's media rows against text + sink + two recent chunks + themselves.
        {"name": "live_media", "kind": "live_media", "text": 77, "audio": 128, "video": 12960, "heads": 24},
    ]


def _spread(rng, low, high):
    """An integer of low..high, even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    while True:
        case = _draw(rng)
        if work(case)["flops"] <= LARGEST_FLOPS:
            return case


def _draw(rng):
    kind = rng.choice(["refine", "causal", "decode", "rope", "dense", "dense", "host", "project", "sparse", "sparse",
                       "live_text", "live_media"])
    # all heads of a model, or one GPU's share of them under sequence parallelism
    heads = rng.choice([3, 6, 7, 12, 14, 24, 28, 56])
    if kind == "refine":
        return {"kind": kind, "rows": _spread(rng, 16, 640), "heads": rng.choice([24, 56])}
    if kind == "causal":
        heads, kv_heads = rng.choice([(8, 2), (16, 16), (16, 8), (28, 4), (32, 8)])
        return {"kind": kind, "rows": _spread(rng, 16, 4096), "heads": heads, "kv_heads": kv_heads}
    if kind == "decode":
        return {"kind": kind, "rows": _spread(rng, 256, 8192), "heads": rng.choice([2, 4, 8, 16])}
    if kind == "rope":
        return {"kind": kind, "rows": _spread(rng, 200, 30000), "heads": heads, "grouped": rng.random() < 0.7}
    if kind == "dense":
        return {"kind": kind, "rows": _spread(rng, 400, 52352), "heads": heads, "sharp": rng.choice([1.0, 2.0, 3.0])}
    if kind == "host":
        return {"kind": kind, "rows": _spread(rng, 1000, 30000), "heads": heads}
    if kind == "project":
        return {"kind": kind, "rows": _spread(rng, 200, 30000), "heads": rng.choice([24, 56])}
    if kind == "sparse":
        return {"kind": kind, "text": _spread(rng, 8, 512), "audio": _spread(rng, 32, 640), "time": rng.randint(6, 37),
                "height": rng.randint(12, 30), "width": rng.randint(20, 54), "heads": heads,
                "alike": rng.random() < 0.5, "fused": rng.random() < 0.5, "kept": rng.choice([0.1, 0.125])}
    if kind == "live_text":
        return {"kind": kind, "rows": _spread(rng, 16, 512), "keys": _spread(rng, 3000, 65000), "heads": heads}
    return {"kind": kind, "text": _spread(rng, 16, 512), "audio": rng.randint(16, 160), "video": _spread(rng, 405, 12960),
            "heads": heads}


# ---- the context a program keeps, and what it holds for one call -----------------------------------

_context = None


def _gpu():
    global _context
    if _context is None:
        torch.cuda.init()
        torch.zeros(1, device="cuda")
        _context = native.Native()
    return _context


class Held:
    """Tensors of a call, their handles, and the library objects to give back with them."""

    def __init__(self, case):
        self.kind, self.gpu, self.handles, self.release, self.keep = case["kind"], _gpu(), [], [], []

    def wrap(self, t, dtype=native.BF16):
        handle = self.gpu.lib.h3b_tensor_wrap(self.gpu.gpu, t.data_ptr(), t.numel(), dtype)
        self.handles.append(handle)
        self.keep.append(t)
        return handle

    def __del__(self):
        for give_back, what in self.release:
            give_back(what)
        for handle in self.handles:
            self.gpu.lib.h3_gpu_tensor_free(handle)


def _normal(g, *shape, sigma=1.0, dtype=torch.bfloat16):
    return (sigma * torch.randn(*shape, generator=g, device="cuda")).to(dtype)


def _unit(g, rows, heads, sharp=1.0):
    """Vectors as the Q/K norm leaves them: unit root mean square, times a gain (queries: how sharp)."""
    x = torch.randn(rows, heads, DIM, generator=g, device="cuda")
    return (x * (sharp * torch.rsqrt(x.square().mean(-1, keepdim=True)))).to(torch.bfloat16)


def _field(g, case):
    """Per token and channel: independent values, or a smooth field over the video grid plus noise."""
    prefix, grid, heads = case["text"] + case["audio"], (case["time"], case["height"], case["width"]), case["heads"]
    if not case["alike"]:
        return torch.randn(prefix + math.prod(grid), heads, DIM, generator=g, device="cuda")
    coarse = torch.randn(1, heads * DIM, *[max(2, -(-n // 6)) for n in grid], generator=g, device="cuda")
    smooth = torch.nn.functional.interpolate(coarse, size=grid, mode="trilinear", align_corners=True)
    video = smooth.reshape(heads * DIM, -1).t().reshape(-1, heads, DIM)
    return torch.cat([torch.randn(prefix, heads, DIM, generator=g, device="cuda"), video])


def _rope_inputs(g, rows):
    angle = 2.0 * math.pi * torch.rand(rows, ROPE_HALF, generator=g, device="cuda")
    weights = [(1.0 + 0.1 * torch.randn(DIM, generator=g, device="cuda")).to(torch.bfloat16) for _ in range(2)]
    return weights + [torch.cos(angle).to(torch.bfloat16), torch.sin(angle).to(torch.bfloat16)]


def _sparse_geometry(case):
    """(tiles, prefix tiles, video tiles each query tile keeps)"""
    prefix = -(-case["text"] // 64) + -(-case["audio"] // 64)
    video = math.prod(-(-case[n] // 4) for n in ("time", "height", "width"))
    return prefix + video, prefix, max(1, math.ceil(case["kept"] * video))


def _rows(case):
    if case["kind"] == "sparse":
        return case["text"] + case["audio"] + case["time"] * case["height"] * case["width"]
    if case["kind"] == "live_media":
        return case["text"] + case["audio"] + case["video"]
    return case["rows"]


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s, kind, heads = Held(case), case["kind"], case["heads"]
    rows, lib, ctx = _rows(case), s.gpu.lib, s.gpu.gpu
    if kind in ("refine", "dense", "causal"):
        q = _unit(g, rows, heads, case.get("sharp", 1.0))
        k = _unit(g, rows, case.get("kv_heads", heads))
        v = _normal(g, rows, case.get("kv_heads", heads), DIM)
        s.out = torch.empty_like(q)
        tensors = [s.wrap(t) for t in (s.out, q, k, v)]
        sizes = (rows, heads, case["kv_heads"]) if kind == "causal" else (rows, heads)
        s.call = {"refine": lib.h3_gpu_sdpa_fa2_bf16, "dense": lib.h3_gpu_sdpa_bf16,
                  "causal": lib.h3_gpu_gqa_causal_bf16}[kind]
        s.args = (ctx, *tensors, *sizes, DIM, SCALE)
    elif kind == "decode":
        q, k, v = (_normal(g, rows, heads, 64, dtype=torch.float16) for _ in range(3))
        s.out = torch.empty_like(q)
        s.call = lib.h3_gpu_sdpa_f16_d64
        s.args = (ctx, *[s.wrap(t, native.F16) for t in (s.out, q, k, v)], rows, heads, 64, 0.125)
    elif kind == "rope":
        qkv = _normal(g, rows, 3 * heads * DIM)
        s.out = [torch.empty(rows, heads, DIM, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
        s.call = lib.h3_gpu_grouped_qkv_rope_bf16 if case["grouped"] else lib.h3_gpu_qkv_rope_bf16
        s.args = (ctx, *[s.wrap(t) for t in [*s.out, qkv, *_rope_inputs(g, rows)]], rows, heads, DIM, ROPE_HALF, EPSILON)
    elif kind == "host":
        q, k = (_unit(g, rows, heads).cpu().pin_memory() for _ in range(2))
        v = _normal(g, rows, heads, DIM).cpu().pin_memory()
        s.out = torch.empty(rows, heads, DIM, dtype=torch.bfloat16, pin_memory=True)
        s.keep += [q, k, v]
        s.call = lib.h3b_sdpa_bf16_host
        s.args = (ctx, *[t.data_ptr() for t in (s.out, q, k, v)], rows, heads, DIM, SCALE, 0)
    elif kind == "project":
        inner = heads * DIM
        residual = _normal(g, rows, HIDDEN)
        x = _normal(g, rows, inner, sigma=0.5)
        weight = _normal(g, HIDDEN, inner, sigma=inner ** -0.5)
        norm = (1.0 + 0.1 * torch.randn(HIDDEN, generator=g, device="cuda")).to(torch.bfloat16)
        modulation = _normal(g, 3, SLOTS, HIDDEN, sigma=0.3)
        # text, audio and video rows have modulation vectors of their own
        row_map = torch.full((rows,), 2, dtype=torch.int32, device="cuda")
        row_map[: rows // 20] = 1
        row_map[: rows // 100] = 0
        s.out = [torch.empty_like(residual) for _ in range(2)]
        tensors = [s.wrap(t) for t in (*s.out, residual, x, weight, norm, modulation, modulation)]
        s.call = lib.h3b_attention_output_gate_adaln_bf16
        s.args = (ctx, *tensors, s.wrap(row_map, native.U32), rows, inner, HIDDEN, SLOTS, 2, 3, 4, EPSILON)
    elif kind == "sparse":
        vsa = s.gpu.call("vsa_new", *[case[n] for n in ("text", "audio", "time", "height", "width")], heads)
        s.release.append((lib.h3_gpu_vsa_free, vsa))
        if not lib.h3b_vsa_set_keep(vsa, _sparse_geometry(case)[2]):
            raise RuntimeError("kept tiles refused")
        field = _field(g, case)
        noise = 0.5 if case["alike"] else 1.0
        qkv = []
        for which in range(3):
            x = torch.randn(rows, heads, DIM, generator=g, device="cuda").mul_(noise)
            if case["alike"]:
                x += field
            if which < 2 and not case["fused"]:
                x *= torch.rsqrt(x.square().mean(-1, keepdim=True))
            qkv.append(x.to(torch.bfloat16))
            del x
        del field
        gate = _normal(g, rows, heads, DIM, sigma=0.3)
        s.out = torch.empty_like(gate)
        if case["fused"]:
            grouped = torch.stack(qkv, dim=2).reshape(rows, 3 * heads * DIM)
            s.call = lib.h3b_vsa_qkv_rope_bf16
            s.args = (vsa, *[s.wrap(t) for t in (s.out, grouped, *_rope_inputs(g, rows), gate)], ROPE_HALF, EPSILON, 1)
        else:
            s.call = lib.h3_gpu_vsa_bf16
            s.args = (vsa, *[s.wrap(t) for t in (s.out, *qkv, gate)])
    elif kind == "live_text":
        q, k = _unit(g, rows, heads), _unit(g, case["keys"], heads)
        v = _normal(g, case["keys"], heads, DIM)
        s.out = torch.empty_like(q)
        s.call = lib.h3_gpu_cross_attention_bf16
        s.args = (ctx, s.wrap(s.out), 0, s.wrap(q), 0, s.wrap(k), s.wrap(v), 0, rows, case["keys"], heads)
    elif kind == "live_media":
        media = case["audio"] + case["video"]
        history = lib.h3b_live_kv_new(ctx, media, heads)
        s.release.append((lib.h3b_live_kv_free, history))
        for _ in range(3):   # sink and two recent chunks: the steady state
            chunk = [s.wrap(t) for t in (_unit(g, media, heads), _normal(g, media, heads, DIM))]
            torch.cuda.synchronize()
            if not (lib.h3b_live_kv_stage(history, *chunk, 0, media, case["audio"]) and lib.h3b_live_kv_commit(history)):
                raise RuntimeError(s.gpu.error())
            s.gpu.submit()
            s.keep.clear()
        q, k = _unit(g, rows, heads), _unit(g, rows, heads)
        v = _normal(g, rows, heads, DIM)
        s.out = torch.zeros(media, heads, DIM, device="cuda", dtype=torch.bfloat16)
        tq, tk, tv = (s.wrap(t) for t in (q, k, v))
        s.stage = (history, tk, tv, case["text"], media, case["audio"])
        s.call = lib.h3b_live_kv_attention_bf16
        s.args = (history, s.wrap(s.out), 0, tq, case["text"], media, tk, tv, case["text"], rows)
    torch.cuda.synchronize()
    return s


def run(state):
    # the clean pass of a live chunk also puts its keys and values into the ring
    if state.kind == "live_media" and not state.gpu.lib.h3b_live_kv_stage(*state.stage):
        raise RuntimeError(state.gpu.error())
    if not state.call(*state.args):
        raise RuntimeError(state.gpu.error())
    return state.out


def work(case):
    kind, heads, rows = case["kind"], case["heads"], _rows(case)
    width = heads * DIM
    if kind in ("refine", "dense", "host"):
        return {"bytes": 4 * rows * width * ADD_BYTES, "flops": 4 * rows * rows * width}
    if kind == "causal":
        return {"bytes": 2 * rows * (heads + case["kv_heads"]) * DIM * ADD_BYTES, "flops": 2 * rows * (rows + 1) * width}
    if kind == "decode":
        return {"bytes": 4 * rows * heads * 64 * ADD_BYTES, "flops": 4 * rows * rows * heads * 64}
    if kind == "rope":
        return {"bytes": 6 * rows * width * ADD_BYTES + 2 * rows * ROPE_HALF * ADD_BYTES, "flops": 20 * rows * width}
    if kind == "project":
        return {"bytes": (rows * width + HIDDEN * width + 3 * rows * HIDDEN) * ADD_BYTES, "flops": 2 * rows * width * HIDDEN}
    if kind == "sparse":
        tiles, prefix, kept = _sparse_geometry(case)
        pairs = prefix * tiles + (tiles - prefix) * (prefix + kept)
        return {"bytes": 5 * rows * width * ADD_BYTES,
                "flops": heads * (pairs * 4 * 64 * 64 * DIM + 4 * tiles * tiles * DIM)}
    if kind == "live_text":
        return {"bytes": 2 * (rows + case["keys"]) * width * ADD_BYTES, "flops": 4 * rows * case["keys"] * width}
    media = case["audio"] + case["video"]
    keys = rows + 2 * media + case["video"]
    return {"bytes": (2 * media + 2 * keys + 2 * media) * width * ADD_BYTES, "flops": 4 * media * keys * width}


def tolerance(case):
    """About four times what each path differs by from the same arithmetic with 64-bit sums (weights
    of an attention row are rounded to the operand type before the second product)."""
    if case["kind"] == "rope":
        return {"rel": 1e-4, "max": 0.05}
    if case["kind"] == "project":
        return {"rel": 4e-4, "max": 0.08}
    if case["kind"] == "decode":
        return {"rel": 1.2e-3, "max": 0.005}
    return {"rel": 1.2e-2, "max": 0.06}
