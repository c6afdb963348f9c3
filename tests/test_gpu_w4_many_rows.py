"""The 4-bit GEMM for more than 16 activation rows: the row-tile kernel's sums are those of the 16-row kernel, bit for bit, at every tile height that its
dispatch can choose, for full and ragged last tiles, all row lengths and formats. The 16-row kernel itself is held to the oracle elsewhere."""
import ctypes as C

import numpy as np
import pytest

from cudapp_b200 import api
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["int4", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("n,k,m", [(128, 768, 17), (256, 1024, 33), (128, 4096, 64), (4096, 768, 65), (8192, 1024, 80), (4096, 2048, 300), (8192, 1024, 511)])
def test_rows_equal_sixteen_row_calls(fmt, n, k, m):
    rng = np.random.default_rng(n + k + m)
    packed = rng.integers(0, 256, (n, k // 2)).astype(np.uint8)
    if fmt == "int4":
        scale = rng.uniform(0.001, 0.01, (n, k // 32)).astype(np.float16).view(np.uint16); up = api.lib.omega_gpu_w4_upload
    elif fmt == "mxfp4":
        scale = rng.integers(118, 124, (n, k // 32)).astype(np.uint8); scale[0, 0] = 0; up = api.lib.omega_gpu_mxfp4_upload
    else:
        scale = rng.integers(0, 80, (n, k // 16)).astype(np.uint8); up = api.lib.omega_gpu_nvfp4_upload
    xb = orc.bf16_bits(rng.normal(0, 1, (m, k)).astype(np.float32))
    t = C.c_void_p()
    assert up(C.c_uint32(n), C.c_uint32(k), packed.ctypes.data_as(C.c_void_p), scale.ctypes.data_as(C.c_void_p), C.byref(t)) == 0, api.last_error()
    rc, y16, y32 = api.w4_gemm_bf16(t, n, xb); assert rc == 0, api.last_error()
    assert np.array_equal(y16, orc.bf16_bits(y32))
    for r in {0, m // 2 // 16 * 16, (m - 1) // 16 * 16}:
        rc, _, part = api.w4_gemm_bf16(t, n, xb[r:r + 16]); assert rc == 0, api.last_error()
        assert np.array_equal(part.view(np.uint32), y32[r:r + 16].view(np.uint32)), r
    api.lib.omega_gpu_w4_free(t)
