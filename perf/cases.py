"""Timed cases of the quantized MoE expert path: the calls a serving process makes, over the sizes it makes them at.

A case is one call of a public entry: the FP8 projections (GEMV, row-table GEMM), the 4-bit GEMM, the FP8 and the 4-bit MoE layer, and the layer
stack. Device cases run on one stream with arguments in device memory, as a serving loop keeps them; host cases give numpy arrays to the drop-in
entries, which stage, run and copy back. Weights are N(0, 0.02) quantised by the format's rule, activations and router logits N(0, 1).
"""
import ctypes as C
import math

import numpy as np
import torch

from cudapp_b200 import api

BF16, U32, VP = torch.bfloat16, C.c_uint32, C.c_void_p
EXPERT_WEIGHTS = 128 * 3 * 2048 * 768           # most weights of one layer: 128 experts, hidden 2048, expert width 768
W4_K = (768, 1024, 2048, 4096)                  # row lengths that every 4-bit format takes
_stream = None


def listed():
    return [
        # the smallest call of the drop-in surface: one projection on one host row (the single-GEMV configuration of the benchmark)
        {"name": "gemv_host_1", "kind": "gemv", "host": True, "groups": 1, "experts": 128, "n": 768, "k": 2048, "bf16": True},
        # gate|up of one token's eight experts, device form: the projection as a decode loop without the layer entry makes it
        {"name": "gemv_top8", "kind": "gemv", "host": False, "groups": 8, "experts": 128, "n": 1536, "k": 2048, "bf16": False},
        # drop-in row-table GEMM on host buffers: 64 tokens x 8 picks, sorted by expert
        {"name": "rows_host_512", "kind": "rows", "host": True, "rows": 512, "experts": 128, "n": 1536, "k": 2048, "bf16": True},
        # dense int4 projection for a decode batch (the W4 configuration of the benchmark)
        {"name": "w4_int4_m16", "kind": "w4", "format": "int4", "m": 16, "n": 4096, "k": 4096},
        # dense NVFP4 projection for a ragged prefill chunk
        {"name": "w4_nvfp4_m300", "kind": "w4", "format": "nvfp4", "m": 300, "n": 4096, "k": 2048},
        # one token through one layer: interactive decode
        {"name": "layer_1", "kind": "layer", "host": False, "tokens": 1, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "exact": True, "shared": False, "skew": 0.0},
        # a decode batch through one layer (the decode-layer configuration)
        {"name": "layer_64", "kind": "layer", "host": False, "tokens": 64, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "exact": True, "shared": False, "skew": 0.0},
        # the same layer called with host arrays
        {"name": "layer_host_256", "kind": "layer", "host": True, "tokens": 256, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "exact": True, "shared": False, "skew": 0.0},
        # a prefill chunk of odd length at the default (exact) activations
        {"name": "layer_1001", "kind": "layer", "host": False, "tokens": 1001, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "exact": True, "shared": False, "skew": 0.5},
        # a long prefill with FP8 activations and skewed load (the prefill configuration)
        {"name": "layer_fp8_4096", "kind": "layer", "host": False, "tokens": 4096, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "exact": False, "shared": False, "skew": 0.5},
        # a decode batch through a layer whose experts are MXFP4
        {"name": "w4layer_mxfp4_64", "kind": "w4layer", "format": "mxfp4", "tokens": 64, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768},
        # a slice of the whole-model decode step: eight layers, 256 tokens, the router inside the stack
        {"name": "stack_router_256", "kind": "stack", "tokens": 256, "layers": 8, "experts": 128, "topk": 8, "hidden": 2048, "inter": 768, "router": True},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _step(rng, lo, hi, step):
    """a multiple of `step` from lo to hi, spread over the logarithm"""
    return _log(rng, lo // step, hi // step) * step


def _experts(rng, hidden, inter):
    most = EXPERT_WEIGHTS // (3 * hidden * inter)
    return min(rng.choice((16, 32, 60, 64, 128)), most)


def draw(rng):
    kind = rng.choice(("gemv", "rows", "w4", "layer", "layer", "layer", "w4layer", "stack"))
    if kind == "gemv":
        n, k = rng.choice(((768, 2048), (1536, 2048), (2048, 768), (_step(rng, 256, 4096, 128), _step(rng, 512, 4096, 128))))
        return {"kind": kind, "host": rng.random() < 0.5, "groups": _log(rng, 1, 64), "experts": 64, "n": n, "k": k, "bf16": rng.random() < 0.5}
    if kind == "rows":
        n, k = rng.choice(((1536, 2048), (2048, 768), (_step(rng, 256, 2048, 128), _step(rng, 512, 2048, 128))))
        return {"kind": kind, "host": rng.random() < 0.5, "rows": _log(rng, 2, 1024), "experts": rng.choice((8, 32, 128)), "n": n, "k": k, "bf16": rng.random() < 0.5}
    if kind == "w4":
        return {"kind": kind, "format": rng.choice(("int4", "mxfp4", "nvfp4")), "m": _log(rng, 1, 512), "n": _step(rng, 768, 8192, 128), "k": rng.choice(W4_K)}
    if kind == "layer":
        hidden, inter = rng.choice(((2048, 768), (2048, 512), (_step(rng, 768, 3072, 256), _step(rng, 256, 768, 128))))
        if hidden * inter > 2048 * 768:
            inter = 2048 * 768 // hidden // 128 * 128
        exact = rng.random() < 0.6
        tokens = _log(rng, 1, 2048) if exact else _log(rng, 16, 4096)
        experts = _experts(rng, hidden, inter)
        return {"kind": kind, "host": rng.random() < 0.2 and tokens <= 512, "tokens": tokens, "experts": experts, "topk": rng.choice((4, 8, 8)), "hidden": hidden, "inter": inter,
                "exact": exact, "shared": rng.random() < 0.2, "skew": rng.choice((0.0, 0.5))}
    if kind == "w4layer":
        hidden, inter = rng.choice(((2048, 768), (2048, 768), (2048, 1024), (1024, 768), (4096, 768)))
        return {"kind": kind, "format": rng.choice(("int4", "mxfp4", "nvfp4")), "tokens": _log(rng, 1, 512), "experts": _experts(rng, hidden, inter), "topk": rng.choice((4, 8)),
                "hidden": hidden, "inter": inter}
    return {"kind": "stack", "tokens": _log(rng, 1, 256), "layers": rng.choice((2, 4, 8)), "experts": rng.choice((32, 64, 128)), "topk": 8, "hidden": 2048, "inter": 768,
            "router": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------- what a program has in hand before the call
def stream():
    """the process's serving stream"""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _ok(rc):
    if rc != 0:
        raise RuntimeError("rc %d: %s" % (rc, api.last_error()))


class State:
    """Handles and buffers of one case; the handles go back to the library with it, last made first."""

    def __init__(self):
        self.handles, self.keep, self.out = [], [], None
        self.run = None

    def own(self, free, handle):
        self.handles.append((free, handle))
        return handle

    def __del__(self):
        while self.handles:
            free, handle = self.handles.pop()
            free(handle)


def _va(t):
    return C.c_uint64(t.data_ptr())


def _device_call(state, fn, *args):
    out = state.out

    def call():
        _ok(fn(*args))
        return out
    state.run = call


def _fp8_tensor(state, g, experts, n, k):
    w8 = torch.empty((experts, n, k), dtype=torch.uint8, device="cuda")
    scale = torch.empty((experts, n // 128, k // 128), dtype=BF16, device="cuda")
    part = max(1, (1 << 27) // (n * k))
    for e in range(0, experts, part):
        m = min(part, experts - e)
        w = (torch.randn((m * n, k), generator=g, device="cuda") * 0.02).to(BF16)
        _ok(api.lib.omega_gpu_fp8_quantize_bf16_dev(U32(m * n), U32(k), _va(w), _va(w8[e]), _va(scale[e])))
    h = VP()
    _ok(api.lib.omega_gpu_fp8_tensor_upload_dev(U32(experts), U32(n), U32(k), _va(w8), _va(scale), C.byref(h)))
    return state.own(api.lib.omega_gpu_fp8_tensor_free, h)


def _e2m1(scaled):
    """nearest E2M1 code of every value"""
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=scaled.device)
    return (torch.bucketize(scaled.abs(), edges, out_int32=True) + (scaled < 0) * 8).to(torch.uint8)


def _w4_tensor(state, g, fmt, n, k):
    packed = torch.empty((n, k // 2), dtype=torch.uint8, device="cuda")
    group = 16 if fmt == "nvfp4" else 32
    scales = torch.empty((n, k // group), dtype=torch.float16 if fmt == "int4" else torch.uint8, device="cuda")
    part = max(1, (1 << 26) // k)
    for r in range(0, n, part):
        w = (torch.randn((min(part, n - r), k), generator=g, device="cuda") * 0.02).view(-1, k // group, group)
        top = w.abs().amax(-1, keepdim=True)
        if fmt == "int4":
            s = (top / 7).to(torch.float16)
            q = (w / s.float()).round_().clamp_(-8, 7).to(torch.int8).bitwise_and_(15).view(torch.uint8)
        elif fmt == "mxfp4":                                          # E8M0: the power of two that puts the largest value at 4 .. 8
            e = torch.floor(torch.log2(top)) - 2
            s = (e + 127).to(torch.uint8)
            q = _e2m1(w / torch.exp2(e))
        else:                                                         # NVFP4: unsigned E4M3 of top / 6
            s = (top / 6).to(torch.float8_e4m3fn)
            q = _e2m1(w / s.float())
            s = s.view(torch.uint8)
        q = q.view(-1, k // 2, 2)
        packed[r:r + part] = q[..., 0] | (q[..., 1] << 4)
        scales[r:r + part] = s.view(-1, k // group)
    upload = {"int4": api.lib.omega_gpu_w4_upload, "mxfp4": api.lib.omega_gpu_mxfp4_upload, "nvfp4": api.lib.omega_gpu_nvfp4_upload}[fmt]
    p, s, h = packed.cpu(), scales.cpu(), VP()
    _ok(upload(U32(n), U32(k), VP(p.data_ptr()), VP(s.data_ptr()), C.byref(h)))
    return state.own(api.lib.omega_gpu_w4_free, h)


def _host_bits(x):
    return x.to(BF16).cpu().view(torch.int16).numpy().view(np.uint16)


def _entries(t, experts):
    tab = np.empty((len(experts), 2), np.int64)
    for i, e in enumerate(experts):
        rc, w, s = api.fp8_tensor_entry(t, int(e))
        _ok(rc)
        tab[i] = w, s
    return torch.from_numpy(tab)


def _prepare_gemv(c, state, g, rng):
    t = _fp8_tensor(state, g, c["experts"], c["n"], c["k"])
    ids = np.sort(rng.choice(c["experts"], c["groups"], replace=False)).astype(np.uint32)
    x = torch.randn((1, c["k"]), generator=g, device="cuda")
    if c["host"]:
        single = api.fp8_gemv_bf16 if c["bf16"] else api.fp8_gemv_f32
        xh = _host_bits(x) if c["bf16"] and c["groups"] == 1 else x.cpu().numpy()     # the grouped host entry takes f32 rows

        def call():
            rc, y = single(t, int(ids[0]), xh) if len(ids) == 1 else api.fp8_gemv_grouped_f32(t, ids, xh)
            _ok(rc)
            return y
        state.run = call
        return
    if c["bf16"]:
        x = x.to(BF16)
    tab = _entries(t, ids).cuda()
    state.out = torch.empty((c["groups"], c["n"]), device="cuda")
    state.keep = [x, tab]
    _device_call(state, api.lib.omega_gpu_fp8_gemv_grouped_async, t, U32(c["groups"]), _va(tab), _va(x), U32(1), C.c_int(int(c["bf16"])), _va(state.out), VP(stream().cuda_stream))


def _prepare_rows(c, state, g, rng):
    t = _fp8_tensor(state, g, c["experts"], c["n"], c["k"])
    M, E = c["rows"], c["experts"]
    tokens = -(-M // 8)
    picks = np.concatenate([rng.permutation(E)[:8] for _ in range(tokens)])[:M]
    order = np.argsort(picks, kind="stable")
    M = len(order)
    ids, rows = picks[order].astype(np.uint32), (order // 8).astype(np.uint32)
    x = torch.randn((tokens, c["k"]), generator=g, device="cuda")
    if c["host"]:
        xh = _host_bits(x) if c["bf16"] else x.cpu().numpy()

        def call():
            rc, y = api.fp8gemm(t, ids, rows, xh)
            _ok(rc)
            return y
        state.run = call
        return
    if c["bf16"]:
        x = x.to(BF16)
    used, first, count = np.unique(ids, return_index=True, return_counts=True)
    seg = torch.zeros((len(used), 4), dtype=torch.int64)
    seg[:, :2] = _entries(t, used)
    seg[:, 2] = torch.from_numpy(first.astype(np.int64) | (count.astype(np.int64) << 32))
    seg, xmap, ymap = seg.cuda(), torch.from_numpy(rows.view(np.int32)).cuda(), torch.from_numpy(order.astype(np.int32)).cuda()
    state.out = torch.empty((M, c["n"]), device="cuda")
    state.keep = [x, seg, xmap, ymap]
    _device_call(state, api.lib.omega_gpu_fp8gemm_async, t, U32(M), U32(len(used)), _va(seg), _va(x), C.c_int(int(c["bf16"])), _va(state.out), _va(xmap), _va(ymap),
                 VP(stream().cuda_stream))


def _prepare_w4(c, state, g, rng):
    t = _w4_tensor(state, g, c["format"], c["n"], c["k"])
    x = torch.randn((c["m"], c["k"]), generator=g, device="cuda").to(BF16)
    state.out = torch.empty((c["m"], c["n"]), dtype=BF16, device="cuda")
    state.keep = [x]
    _device_call(state, api.lib.omega_gpu_w4_gemm_async, t, U32(c["m"]), _va(x), _va(state.out), C.c_uint64(0), VP(stream().cuda_stream))


def _layer(c, state, g, max_tokens):
    E = c["experts"] + int(c.get("shared", False))
    gate_up, down = _fp8_tensor(state, g, E, 2 * c["inter"], c["hidden"]), _fp8_tensor(state, g, E, c["hidden"], c["inter"])
    pieces = {} if c.get("exact", True) else {"x_pieces": 1, "act_pieces": 1}
    rc, layer = api.moe_layer_create(gate_up, down, topk=c["topk"], max_tokens=max_tokens, shared_expert=c.get("shared", False), **pieces)
    _ok(rc)
    return state.own(api.lib.omega_gpu_moe_layer_free, layer)


def _activations(c, g, layers=1):
    logits = torch.randn((layers, c["tokens"], c["experts"]), generator=g, device="cuda")
    if c.get("skew"):
        logits += torch.randn(c["experts"], generator=g, device="cuda") * c["skew"]
    return logits.to(BF16), torch.randn((c["tokens"], c["hidden"]), generator=g, device="cuda").to(BF16)


def _outputs(c, state):
    state.out = (torch.empty((c["tokens"], c["hidden"]), device="cuda"), torch.empty((c["tokens"], c["hidden"]), dtype=BF16, device="cuda"))
    return _va(state.out[0]), _va(state.out[1])


def _prepare_layer(c, state, g, rng):
    layer = _layer(c, state, g, c["tokens"])
    logits, x = _activations(c, g)
    if c["host"]:
        lh, xh, slots = _host_bits(logits[0]), _host_bits(x), c["topk"] + int(c["shared"])

        def call():
            rc, o16, o32, ids, wts = api.moe_layer_bf16(layer, lh, xh, topk=slots)
            _ok(rc)
            return o32, torch.from_numpy(o16.view(np.int16)).view(BF16), ids, wts
        state.run = call
        return
    state.keep = [logits, x]
    _device_call(state, api.lib.omega_gpu_moe_layer_async, layer, U32(c["tokens"]), _va(logits), _va(x), *_outputs(c, state), VP(stream().cuda_stream))


def _prepare_w4layer(c, state, g, rng):
    E, H, I = c["experts"], c["hidden"], c["inter"]
    gate_up, down, layer = _w4_tensor(state, g, c["format"], E * 2 * I, H), _w4_tensor(state, g, c["format"], E * H, I), VP()
    _ok(api.lib.omega_gpu_moe_w4_layer_create(gate_up, down, U32(E), U32(c["topk"]), U32(c["tokens"]), C.c_int(1), C.byref(layer)))
    state.own(api.lib.omega_gpu_moe_w4_layer_free, layer)
    logits, x = _activations(c, g)
    state.keep = [logits, x]
    _device_call(state, api.lib.omega_gpu_moe_w4_layer_async, layer, U32(c["tokens"]), _va(logits), _va(x), *_outputs(c, state), VP(stream().cuda_stream))


def _prepare_stack(c, state, g, rng):
    layers = [_layer(c, state, g, c["tokens"]) for _ in range(c["layers"])]
    rc, stack = api.moe_stack_create(layers)
    _ok(rc)
    state.own(api.lib.omega_gpu_moe_stack_free, stack)
    logits, x = _activations(c, g, c["layers"])
    if c["router"]:
        for i in range(c["layers"]):
            gate = torch.randn((c["experts"], c["hidden"]), generator=g, device="cuda") * 0.02
            norm = 1 + 0.1 * torch.randn(c["hidden"], generator=g, device="cuda")
            rc, router = api.moe_router_create(_host_bits(gate), norm.cpu().numpy())
            _ok(rc)
            state.handles.insert(0, (api.lib.omega_gpu_moe_router_free, router))     # outlives the stack
            _ok(api.lib.omega_gpu_moe_stack_set_router(stack, U32(i), router))
    state.keep = [logits, x]
    _device_call(state, api.lib.omega_gpu_moe_stack_async, stack, U32(c["tokens"]), C.c_uint64(0 if c["router"] else logits.data_ptr()), _va(x), *_outputs(c, state),
                 VP(stream().cuda_stream))


def prepare(case, seed):
    state = State()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    {"gemv": _prepare_gemv, "rows": _prepare_rows, "w4": _prepare_w4, "layer": _prepare_layer, "w4layer": _prepare_w4layer,
     "stack": _prepare_stack}[case["kind"]](case, state, g, np.random.default_rng(seed))
    torch.cuda.synchronize()                                          # inputs were made on torch's own stream
    return state


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _fp8_bytes(n, k):
    return n * k + (n // 128) * (k // 128) * 4


def _w4_bytes(fmt, n, k):
    return n * k // 2 + n * (k // (16 if fmt == "nvfp4" else 32)) * (2 if fmt == "int4" else 1)


def _distinct(experts, topk, tokens):
    """experts that `tokens` tokens with `topk` different picks each are expected to reach"""
    return experts * (1.0 - (1.0 - min(1.0, topk / experts)) ** tokens)


def work(case):
    c = case
    if c["kind"] in ("gemv", "rows"):
        rows = c.get("groups") or c["rows"]
        used = rows if c["kind"] == "gemv" else _distinct(c["experts"], min(8, rows, c["experts"]), -(-rows // 8))
        x_rows = 1 if c["kind"] == "gemv" else -(-rows // 8)
        return {"bytes": used * _fp8_bytes(c["n"], c["k"]) + x_rows * c["k"] * (2 if c["bf16"] else 4) + rows * c["n"] * 4, "flops": 2.0 * rows * c["n"] * c["k"]}
    if c["kind"] == "w4":
        return {"bytes": _w4_bytes(c["format"], c["n"], c["k"]) + 2 * c["m"] * (c["n"] + c["k"]), "flops": 2.0 * c["m"] * c["n"] * c["k"]}
    T, E, H, I, layers = c["tokens"], c["experts"], c["hidden"], c["inter"], c.get("layers", 1)
    shared = int(c.get("shared", False))
    if c["kind"] == "w4layer":
        expert = _w4_bytes(c["format"], 2 * I, H) + _w4_bytes(c["format"], H, I)
    else:
        expert = _fp8_bytes(2 * I, H) + _fp8_bytes(H, I)
    flops = 2.0 * layers * T * (c["topk"] + shared) * 3 * H * I
    routing = 2 * E * T
    if c.get("router"):
        routing = 2 * E * H + 4 * H
        flops += 2.0 * layers * T * E * H
    return {"bytes": layers * ((_distinct(E, c["topk"], T) + shared) * expert + routing) + T * H * (2 + 4 + 2), "flops": flops}


def tolerance(case):
    if case["kind"] in ("gemv", "rows"):
        return {"rel": 1e-5}                                          # f32 sums of exact products
    if case["kind"] == "layer" and not case["exact"]:
        return {"rel": 1e-2}                                          # FP8 activations: a sum's last bit can move a value to the next code
    return {"rel": 4e-3, "max": 0.05}                                 # bf16 results
