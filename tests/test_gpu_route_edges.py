"""Top-k and plan in one launch (up to 32 tokens) give the picks, weights and results of the two kernels that larger calls take: the tokens of a 40-token call
repeated in calls around the limit, with and without a shared expert, at an expert count whose shared memory only leaves room for fewer tokens, and at those
where the dynamic shared memory of some call (239: 32 tokens, 254: 29, 259 and a shared one: 28) comes to 48 KB less the kernel's few static bytes."""
import numpy as np
import pytest

from cudapp_b200 import api
from oracle import oracle as orc
from tests.test_gpu_ops import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,shared", [(16, False), (17, True), (256, False), (239, False), (254, False), (260, True)])
def test_small_calls_route_like_large_ones(E, shared):
    rng = np.random.default_rng(E)
    H, I, K, T = 256, 128, 4, 40
    wgu, sgu = make_weights(rng, E, 2 * I, H); wdn, sdn = make_weights(rng, E, H, I)
    rc, tgu = api.fp8_tensor_upload(E, 2 * I, H, wgu, sgu); assert rc == 0, api.last_error()
    rc, tdn = api.fp8_tensor_upload(E, H, I, wdn, sdn); assert rc == 0, api.last_error()
    logits = orc.bf16_bits(np.round(rng.normal(0, 1, (T, E - shared)), 1).astype(np.float32))     # rounded: ties
    x = orc.bf16_bits(rng.normal(0, 1, (T, H)).astype(np.float32))
    rc, layer = api.moe_layer_create(tgu, tdn, topk=K, max_tokens=T, shared_expert=shared); assert rc == 0, api.last_error()
    rc, _, o32, ids, w = api.moe_layer_bf16(layer, logits, x, topk=K + shared); assert rc == 0, api.last_error()
    for t in (1, 9, 27, 28, 29, 30, 31, 32, 33):
        rc, _, p32, pids, pw = api.moe_layer_bf16(layer, logits[:t], x[:t], topk=K + shared); assert rc == 0, api.last_error()
        assert np.array_equal(pids, ids[:t]) and np.array_equal(pw.view(np.uint32), w[:t].view(np.uint32))
        assert np.array_equal(p32.view(np.uint32), o32[:t].view(np.uint32))                       # a row's sums do not depend on its neighbours
    api.lib.omega_gpu_moe_layer_free(layer); api.fp8_tensor_free(tgu); api.fp8_tensor_free(tdn)
