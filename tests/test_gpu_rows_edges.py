"""The exact row kernel and the host result paths where their shapes change: rows per pass (8, or 4 past k = 2048), x resident (up to k = 4096) or staged by
chunks past it, one turn or several per CTA, the three lane widths, and results around the size that is stored straight into host memory. Oracle: the reference
kernels' own summation order, bit for bit."""
import numpy as np
import pytest

from cudapp_b200 import api
from oracle import oracle as orc
from tests.test_gpu_ops import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(128, 128), (256, 256), (384, 2048), (128, 2560), (128, 4096), (128, 4224), (256, 8192)])
@pytest.mark.parametrize("bf16", [False, True])
def test_row_table_edges(n, k, bf16):
    rng = np.random.default_rng(n + k)
    counts = [1, 0, 2, 7, 8, 9, 17]                                    # around one and two passes of four and of eight rows
    w8, sc = make_weights(rng, len(counts), n, k)
    rc, t = api.fp8_tensor_upload(len(counts), n, k, w8, sc); assert rc == 0, api.last_error()
    ids = np.repeat(np.arange(len(counts), dtype=np.uint32), counts)
    xb = orc.bf16_bits(rng.normal(0, 1, (11, k)).astype(np.float32)); x = orc.bf16_to_f32(xb)
    rows = rng.integers(0, 11, len(ids)).astype(np.uint32)
    rc, y = api.fp8gemm(t, ids, rows, xb if bf16 else x); assert rc == 0, api.last_error()
    for i in range(len(ids)):
        assert np.array_equal(y[i].view(np.uint32), orc.gemv_emu(w8[ids[i]], sc[ids[i]], x[rows[i]]).view(np.uint32)), (i, ids[i])
    api.fp8_tensor_free(t)


@pytest.mark.parametrize("groups", [1, 8, 9, 63, 64, 65, 700])
def test_grouped_gemv_result_sizes(groups):
    """[groups, 128] f32 results: 64 groups are exactly the 32 KB that the kernel stores itself, 700 go through two staging chunks where the caller's array is pageable"""
    rng = np.random.default_rng(groups)
    E, n, k = 6, 128, 512
    w8, sc = make_weights(rng, E, n, k)
    rc, t = api.fp8_tensor_upload(E, n, k, w8, sc); assert rc == 0, api.last_error()
    ids = rng.integers(0, E, groups).astype(np.uint32); x = rng.normal(0, 1, (groups, k)).astype(np.float32)
    want = np.stack([orc.gemv_emu(w8[e], sc[e], x[g]) for g, e in enumerate(ids)])
    kept = []
    for _ in range(3):                                                 # results of earlier calls stay what they were
        rc, y = api.fp8_gemv_grouped_f32(t, ids, x); assert rc == 0, api.last_error()
        kept.append(y)
    pageable = np.empty((groups, n), np.float32)
    rc = api.lib.omega_gpu_fp8_gemv_grouped_f32(t, api.C.c_uint32(groups), api._p(ids), api._p(x), api.C.c_uint32(groups), api._p(pageable), None); assert rc == 0, api.last_error()
    for y in kept + [pageable]:
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    api.fp8_tensor_free(t)


@pytest.mark.parametrize("k", [128, 640, 2304, 3968, 4096, 4224, 8192, 8320])
def test_gemv_row_lengths(k):
    """one row per warp (few groups) and four (many, or a CTA budget, where a CTA also makes several turns); x resident up to k = 4096 and by chunks past it;
    all lane widths, fewer K steps than are prefetched, and remainders of them"""
    rng = np.random.default_rng(k)
    E, n = 3, 256
    w8, sc = make_weights(rng, E, n, k)
    rc, t = api.fp8_tensor_upload(E, n, k, w8, sc); assert rc == 0, api.last_error()
    x = rng.normal(0, 1, (24, k)).astype(np.float32)
    for groups, budget in ((1, 0), (2, 0), (18, 0), (19, 0), (24, 0), (2, 1), (2, 3), (24, 5)):
        ids = rng.integers(0, E, groups).astype(np.uint32)
        api.lib.omega_gpu_fp8_set_cta_budget(api.C.c_uint32(budget))
        try:
            rc, y = api.fp8_gemv_grouped_f32(t, ids, x[:groups]); assert rc == 0, api.last_error()
        finally:
            api.lib.omega_gpu_fp8_set_cta_budget(api.C.c_uint32(0))
        for g, e in enumerate(ids):
            assert np.array_equal(y[g].view(np.uint32), orc.gemv_emu(w8[e], sc[e], x[g]).view(np.uint32)), (groups, budget, g)
    xb = orc.bf16_bits(x[0])
    rc, y = api.fp8_gemv_bf16(t, 1, xb); assert rc == 0, api.last_error()
    assert np.array_equal(y.view(np.uint32), orc.gemv_emu(w8[1], sc[1], orc.bf16_to_f32(xb)).view(np.uint32))
    api.fp8_tensor_free(t)


@pytest.mark.parametrize("k", [640, 2048, 2304, 4224, 8192])
def test_row_table_turns(k):
    """96 segments of [512, k]: a CTA makes two turns over weight groups, so weights are fetched across turns and, past k = 4096, x is staged anew in the second;
    segments of one, two and three passes among them"""
    rng = np.random.default_rng(k)
    E, n = 96, 512
    w8 = rng.integers(0, 256, (E, n, k), dtype=np.uint8); w8[(w8 & 0x7f) == 0x7f] = 0
    sc = rng.integers(0x3b00, 0x3c00, (E, n // 128, k // 128)).astype(np.uint16)
    rc, t = api.fp8_tensor_upload(E, n, k, w8, sc); assert rc == 0, api.last_error()
    counts = np.ones(E, np.int64); counts[5::16] = 4; counts[9::32] = 9; counts[20::48] = 17
    ids = np.repeat(np.arange(E, dtype=np.uint32), counts)
    xb = orc.bf16_bits(rng.normal(0, 1, (13, k)).astype(np.float32)); x = orc.bf16_to_f32(xb)
    rows = rng.integers(0, 13, len(ids)).astype(np.uint32)
    info = api.Fp8GemmInfo()
    rc, y = api.fp8gemm(t, ids, rows, xb if k % 512 else x, info); assert rc == 0, api.last_error()
    assert info.grid_x * 16 < n                                        # several turns
    for i in range(len(ids)):
        assert np.array_equal(y[i].view(np.uint32), orc.gemv_emu(w8[ids[i]], sc[ids[i]], x[rows[i]]).view(np.uint32)), (i, ids[i])
    api.fp8_tensor_free(t)
