"""Weight gradients of the warm-start net on the tensor cores (unet_dw.cu) on
grids whose levels are thin, odd in units of the K-tile, or shorter than one
tile row: against the CPU reference network, layer by layer, with the bound
that BF16 storage sets (as for the cubic grid in test_gpu_unet.py)."""
import ctypes as C

import numpy as np
import pytest

from picfoam_gb300 import abi, native
from test_gpu_unet import F64P, f32p, make_net, unet_sample

pytestmark = pytest.mark.gpu

LAYERS = [(2, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16), (16, 1)]


@pytest.mark.parametrize("X, Y, Z", [(8, 32, 32), (64, 16, 8), (40, 16, 64), (4, 4, 512)])
def test_weight_gradients_match_reference(gpu, oracle_backend, X, Y, Z):
    lib, olib = native.load(), oracle_backend.load()
    V = X * Y * Z
    h = make_net(lib, X, Y, Z, seed=X + Y)
    try:
        n = lib.picgpu_unet_param_count()
        w = np.zeros(n, np.float32)
        assert lib.picgpu_unet_get_weights(h, f32p(w)) == abi.OK
        x, t, m = unet_sample(np.random.default_rng(X), V)
        g, again = np.zeros(n, np.float32), np.zeros(n, np.float32)
        loss = C.c_double()
        for out in (g, again):
            assert lib.picgpu_unet_gradients(h, f32p(x), f32p(t), f32p(m), f32p(out), C.byref(loss)) == abi.OK
        gref, gexact = np.zeros(n), np.zeros(n)
        for emulate, out in ((1, gref), (0, gexact)):
            assert olib.oracle_unet_gradients(X, Y, Z, f32p(w), f32p(x), f32p(t), f32p(m), emulate,
                                              out.ctypes.data_as(F64P), None) == 0
        off = 0
        for ci, co in LAYERS:
            s = slice(off, off + 27 * ci * co)
            off = s.stop
            bf16_effect = np.linalg.norm(gexact[s] - gref[s]) / np.linalg.norm(gexact[s])
            assert np.linalg.norm(g[s] - gref[s]) <= (1.5 * bf16_effect + 5e-3) * np.linalg.norm(gref[s]), (ci, co)
            # the sums of the position ranges meet in FP32, in any order
            assert np.linalg.norm(g[s] - again[s]) <= 1e-5 * np.linalg.norm(g[s]), (ci, co)
    finally:
        lib.picgpu_unet_destroy(h)
