"""Buffers of the host entries in every kind of memory: pageable, page-locked and device memory give the same bits, below and above the sizes where the copies
change their way (64 KB to the device, 32 KB back, 256 KB staging chunks)."""
import ctypes as C

import numpy as np
import pytest

from cudapp_b200 import api
from oracle import oracle as orc
from tests.test_gpu_ops import make_weights

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr())


def in_memory(a, kind):
    """`a` as a torch tensor (bits kept) in that kind of memory"""
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy())
    return t.pin_memory() if kind == "page-locked" else t.cuda() if kind == "device" else t


@pytest.fixture(scope="module")
def tensors():
    rng = np.random.default_rng(5)
    E, H, I = 8, 512, 256
    wgu, sgu = make_weights(rng, E, 2 * I, H); wdn, sdn = make_weights(rng, E, H, I)
    rc, gu = api.fp8_tensor_upload(E, 2 * I, H, wgu, sgu); assert rc == 0, api.last_error()
    rc, dn = api.fp8_tensor_upload(E, H, I, wdn, sdn); assert rc == 0, api.last_error()
    yield E, H, I, gu, dn
    api.fp8_tensor_free(gu); api.fp8_tensor_free(dn)


@pytest.mark.parametrize("kind", ["page-locked", "device"])
@pytest.mark.parametrize("rows", [16, 300])
def test_row_table_input(tensors, rows, kind):
    import torch
    E, H, I, gu, _ = tensors
    rng = np.random.default_rng(rows)
    ids = np.sort(rng.integers(0, E, rows)).astype(np.uint32); tok = np.arange(rows, dtype=np.uint32)
    x = rng.normal(0, 1, (rows, H)).astype(np.float32)                       # 32 KB, 600 KB
    rc, want = api.fp8gemm(gu, ids, tok, x); assert rc == 0, api.last_error()
    xt = in_memory(x, kind); torch.cuda.synchronize()
    y = np.empty_like(want)
    rc = api.lib.omega_gpu_fp8gemm_f32(gu, C.c_uint32(rows), api._p(ids), api._p(tok), ptr(xt), C.c_uint32(rows), api._p(y), None); assert rc == 0, api.last_error()
    assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("kind", ["pageable", "page-locked", "device"])
@pytest.mark.parametrize("tokens", [4, 1100])
def test_layer_buffers(tensors, tokens, kind):
    """every buffer of the layer's host entry; 1100 tokens: 1.1 MB of x, 2.2 MB of results (more than the staging ring holds at once)"""
    import torch
    E, H, I, gu, dn = tensors
    rng = np.random.default_rng(tokens)
    logits = orc.bf16_bits(rng.normal(0, 1, (tokens, E)).astype(np.float32)); x = orc.bf16_bits(rng.normal(0, 1, (tokens, H)).astype(np.float32))
    rc, layer = api.moe_layer_create(gu, dn, topk=2, max_tokens=tokens); assert rc == 0, api.last_error()
    rc, *want = api.moe_layer_bf16(layer, logits, x, topk=2); assert rc == 0, api.last_error()
    lt, xt = in_memory(logits, kind), in_memory(x, kind)
    out = [in_memory(np.zeros_like(a), kind) for a in want[:2]]
    ids, w = np.empty((tokens, 2), np.uint32), np.empty((tokens, 2), np.float32)
    torch.cuda.synchronize()
    rc = api.lib.omega_gpu_moe_layer_bf16(layer, C.c_uint32(tokens), ptr(lt), ptr(xt), ptr(out[0]), ptr(out[1]), api._p(ids), api._p(w)); assert rc == 0, api.last_error()
    for got, ref in zip(out, want):
        assert np.array_equal(got.cpu().numpy().view(ref.dtype).reshape(ref.shape), ref)
    assert np.array_equal(ids, want[2]) and np.array_equal(w, want[3])
    api.lib.omega_gpu_moe_layer_free(layer)


@pytest.mark.parametrize("kind", ["pageable", "page-locked"])
@pytest.mark.parametrize("rows", [1, 16, 17, 300, 1100])
def test_refused_result_is_left_alone(rows, kind):
    """a word that equals the poison refuses the call, whatever the size of the result (16 rows: the last that the kernel stores itself), and y is as it was"""
    E, n, k = 2, 512, 256
    w8 = np.zeros((E, n, k), np.uint8); w8[1, 100, 0] = 0x38                   # one weight of 1
    rc, t = api.fp8_tensor_upload(E, n, k, w8, np.full((E, n // 128, k // 128), 0x3f80, np.uint16)); assert rc == 0, api.last_error()
    x = np.ones((rows, k), np.float32); x[rows // 2, 0] = -999.0
    ids, tok = np.full(rows, 1, np.uint32), np.arange(rows, dtype=np.uint32)
    y = in_memory(np.full((rows, n), 7, np.float32), kind)
    rc = api.lib.omega_gpu_fp8gemm_f32(t, C.c_uint32(rows), api._p(ids), api._p(tok), api._p(x), C.c_uint32(rows), ptr(y), None)
    assert rc == api.CHIP_FAIL and "poison" in api.last_error()
    assert (y.numpy().view(np.float32) == 7).all()
    x[rows // 2, 0] = 3                                                        # and the next call is served
    rc = api.lib.omega_gpu_fp8gemm_f32(t, C.c_uint32(rows), api._p(ids), api._p(tok), api._p(x), C.c_uint32(rows), ptr(y), None); assert rc == 0, api.last_error()
    want = np.zeros((rows, n), np.float32); want[:, 100] = x[:, 0]
    assert np.array_equal(y.numpy().view(np.float32).reshape(rows, n), want)
    api.fp8_tensor_free(t)


def test_kept_results(tensors):
    """results kept past what the binding page-locks: later ones lie in ordinary memory and all of them stay what they were"""
    E, H, I, gu, _ = tensors
    rng = np.random.default_rng(9)
    ids = np.sort(rng.integers(0, E, 64)).astype(np.uint32); tok = np.arange(64, dtype=np.uint32)
    x = [rng.normal(0, 1, (64, H)).astype(np.float32) for _ in range(12)]
    kept = []
    for v in x:                                                                # 128 KB each
        rc, y = api.fp8gemm(gu, ids, tok, v); assert rc == 0, api.last_error()
        kept.append(y)
    before = api._pool.blocks[128 << 10]
    assert before <= api.POOL_BLOCKS < len(kept) and api._pool.held <= api.POOL_BYTES
    for v, y in zip(x, kept):
        for r in (0, 31, 63):
            rc, one = api.fp8gemm(gu, ids[r:r + 1], tok[:1], v[r:r + 1]); assert rc == 0, api.last_error()
            assert np.array_equal(one[0].view(np.uint32), y[r].view(np.uint32))


def test_result_that_takes_long(tensors):
    """a small result is waited for in host memory for 2 ms at most and by the stream past that: a call behind work that fills the device for longer"""
    import torch
    E, H, I, gu, _ = tensors
    x = np.random.default_rng(11).normal(0, 1, H).astype(np.float32)
    rc, want = api.fp8_gemv_f32(gu, 3, x); assert rc == 0, api.last_error()
    a, b = (torch.randn((8192, 8192), device="cuda") for _ in range(2))
    torch.mm(a, b); torch.cuda.synchronize()
    for _ in range(4):
        torch.mm(a, b)                                                         # about 20 ms each in f32
    rc, got = api.fp8_gemv_f32(gu, 3, x); assert rc == 0, api.last_error()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    torch.cuda.synchronize()
