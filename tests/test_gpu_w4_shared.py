"""4-bit tensors shared by several layers: each layer keeps its own shape, so a smaller layer made later, or a shape set for the grouped GEMM entry, changes nothing
for the ones before."""
import ctypes as C

import numpy as np
import pytest

from cudapp_b200 import api
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
U32 = C.c_uint32


def run(layer, logits, x):
    T, H = x.shape
    out = np.empty((T, H), np.float32)
    rc = api.lib.omega_gpu_moe_w4_layer_bf16(layer, U32(T), api._p(logits), api._p(x), None, api._p(out), None, None); assert rc == 0, api.last_error()
    return out


def test_layers_on_the_same_tensors():
    rng = np.random.default_rng(3)
    E, H, I, K, T = 4, 768, 768, 2, 256
    def tensor(n, k):
        t = C.c_void_p(); packed = rng.integers(0, 256, (n, k // 2)).astype(np.uint8); scale = rng.integers(118, 122, (n, k // 32)).astype(np.uint8)
        assert api.lib.omega_gpu_mxfp4_upload(U32(n), U32(k), api._p(packed), api._p(scale), C.byref(t)) == 0, api.last_error()
        return t
    gu, dn = tensor(E * 2 * I, H), tensor(E * H, I)
    def make(tokens):
        h = C.c_void_p()
        assert api.lib.omega_gpu_moe_w4_layer_create(gu, dn, U32(E), U32(K), U32(tokens), C.c_int(1), C.byref(h)) == 0, api.last_error()
        return h
    logits = orc.bf16_bits(rng.normal(0, 1, (T, E)).astype(np.float32)); x = orc.bf16_bits(rng.normal(0, 1, (T, H)).astype(np.float32))
    large = make(T)
    want = run(large, logits, x)
    small = make(1)                                                   # room for 12 row tiles; 256 tokens need over 30
    def again(order):                                                  # other tokens in every row than the call before: nothing left over can pass for a result
        assert np.array_equal(run(large, np.ascontiguousarray(logits[order]), np.ascontiguousarray(x[order])).view(np.uint32), want[order].view(np.uint32))
    again(np.arange(T)[::-1])
    assert np.array_equal(run(small, logits[7:8], x[7:8]).view(np.uint32), want[7:8].view(np.uint32))
    assert api.lib.omega_gpu_w4_reserve_grouped(dn, U32(H), U32(1)) == 0
    again(np.roll(np.arange(T), 5))
    for free, h in ((api.lib.omega_gpu_moe_w4_layer_free, small), (api.lib.omega_gpu_moe_w4_layer_free, large), (api.lib.omega_gpu_w4_free, gu), (api.lib.omega_gpu_w4_free, dn)):
        free(h)
