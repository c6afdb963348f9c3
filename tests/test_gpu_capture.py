"""The stream-ordered entries inside a caller's own CUDA graph: their kernels are launched as programmatic dependents of one another, which a capture records as
edges. A replay on new inputs, with the caller's work before, between and after them and another stream joined in, gives the bits of plain calls."""
import ctypes as C

import numpy as np
import pytest

from cudapp_b200 import api
from tests.test_gpu_layer import build_layer, free_layer

pytestmark = pytest.mark.gpu
U32 = C.c_uint32


def va(t):
    return C.c_uint64(t.data_ptr())


def here():
    import torch
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def ok(rc):
    assert rc == 0, api.last_error()


def compare(call, inputs, fill, scratch):
    """`call` three times in one graph (once behind a join with another stream), replayed twice on new inputs, against calls without a graph"""
    import torch
    side, s = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        fill(inputs, 0); call()                                                 # attributes and allocations are made outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        scratch.add_(1)
        first = [t.clone() for t in call()]
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            inputs[-1].add_(0)                                                  # the next call's input is (re)written on the other stream
        torch.cuda.current_stream().wait_stream(side)
        second = [t.clone() for t in call()]
        third = call()                                                          # back to back: the chain runs from one call into the next
        scratch.add_(1)
    for seed in (1, 2):
        with torch.cuda.stream(s):
            fill(inputs, seed)
            want = [t.clone() for t in call()]
            for t in third:
                t.zero_()
            g.replay()
        torch.cuda.synchronize()
        for got in (first, second, third):
            for a, b in zip(got, want):
                assert torch.equal(a.view(torch.int32), b.view(torch.int32)) if a.dtype == torch.float32 else torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert (scratch == 4).all()
    del g


def fill_bf16(inputs, seed):
    import torch
    gen = torch.Generator(device="cuda"); gen.manual_seed(seed)
    for t in inputs:
        t.copy_(torch.randn(t.shape, generator=gen, device="cuda"))


@pytest.mark.parametrize("engine,tokens", [(api.ENGINE_MMA, 1), (api.ENGINE_MMA, 40), (api.ENGINE_MMA, 600), (api.ENGINE_FMA, 3), (api.ENGINE_FMA, 40)])
def test_layer(engine, tokens):
    import torch
    E, H, I, K = 16, 512, 256, 4
    m = build_layer(np.random.default_rng(tokens), E, H, I, tokens, engine, K)
    bf = dict(dtype=torch.bfloat16, device="cuda")
    logits, x = torch.empty((tokens, E), **bf), torch.empty((tokens, H), **bf)
    out = (torch.empty((tokens, H), device="cuda"), torch.empty((tokens, H), **bf))

    def call():
        ok(api.lib.omega_gpu_moe_layer_async(m["layer"], U32(tokens), va(logits), va(x), va(out[0]), va(out[1]), here()))
        return out
    compare(call, [logits, x], fill_bf16, torch.zeros(4, device="cuda"))
    free_layer(m)


def upload_mxfp4(rng, n, k):
    t = C.c_void_p(); packed = rng.integers(0, 256, (n, k // 2)).astype(np.uint8); scale = rng.integers(116, 122, (n, k // 32)).astype(np.uint8)
    ok(api.lib.omega_gpu_mxfp4_upload(U32(n), U32(k), api._p(packed), api._p(scale), C.byref(t)))
    return t


@pytest.mark.parametrize("m", [1, 16, 17, 300])
def test_four_bit_gemm(m):
    import torch
    n, k = 512, 1024
    t = upload_mxfp4(np.random.default_rng(m), n, k)
    x, y = torch.empty((m, k), dtype=torch.bfloat16, device="cuda"), torch.empty((m, n), dtype=torch.bfloat16, device="cuda")

    def call():
        ok(api.lib.omega_gpu_w4_gemm_async(t, U32(m), va(x), va(y), C.c_uint64(0), here()))
        return (y,)
    compare(call, [x], fill_bf16, torch.zeros(4, device="cuda"))
    api.lib.omega_gpu_w4_free(t)


@pytest.mark.parametrize("tokens", [1, 33])
def test_four_bit_layer(tokens):
    import torch
    E, H, I, K = 8, 768, 768, 2
    rng = np.random.default_rng(tokens)
    gu, dn, layer = upload_mxfp4(rng, E * 2 * I, H), upload_mxfp4(rng, E * H, I), C.c_void_p()
    ok(api.lib.omega_gpu_moe_w4_layer_create(gu, dn, U32(E), U32(K), U32(tokens), C.c_int(1), C.byref(layer)))
    bf = dict(dtype=torch.bfloat16, device="cuda")
    logits, x = torch.empty((tokens, E), **bf), torch.empty((tokens, H), **bf)
    out = (torch.empty((tokens, H), device="cuda"), torch.empty((tokens, H), **bf))

    def call():
        ok(api.lib.omega_gpu_moe_w4_layer_async(layer, U32(tokens), va(logits), va(x), va(out[0]), va(out[1]), here()))
        return out
    compare(call, [logits, x], fill_bf16, torch.zeros(4, device="cuda"))
    for free, h in ((api.lib.omega_gpu_moe_w4_layer_free, layer), (api.lib.omega_gpu_w4_free, gu), (api.lib.omega_gpu_w4_free, dn)):
        free(h)


def test_gemv():
    import torch
    rng = np.random.default_rng(8)
    E, n, k = 4, 256, 640
    w8 = rng.integers(0, 0x70, (E, n, k)).astype(np.uint8); sc = np.full((E, n // 128, k // 128), 0x3c00, np.uint16)
    rc, t = api.fp8_tensor_upload(E, n, k, w8, sc); ok(rc)
    tab = torch.tensor([api.fp8_tensor_entry(t, e)[1:] for e in (3, 0, 2)], dtype=torch.int64, device="cuda")
    x, y = torch.empty((3, k), device="cuda"), torch.empty((3, n), device="cuda")

    def call():
        ok(api.lib.omega_gpu_fp8_gemv_grouped_async(t, U32(3), va(tab), va(x), U32(3), C.c_int(0), va(y), here()))
        return (y,)
    compare(call, [x], fill_bf16, torch.zeros(4, device="cuda"))
    api.fp8_tensor_free(t)
