"""The tensor-core weight gradient of each layer of the warm-start net against
64-bit sums of the same operands.  The products of BF16 values are exact and the
FP32 operands go in as three BF16 parts, so what is left is the rounding of the
sums: 16 truncated additions in the tensor core, then FP32 sums of those.  The
bound is 8 ulps of FP32 (2^-23 each) of the gradient's norm; without the third
part of an FP32 operand it would be 2^-16, with sums left in the tensor core over
the whole grid 2.5e-6 and more."""
import ctypes as C

import numpy as np
import pytest

from picfoam_gb300 import abi, native

pytestmark = pytest.mark.gpu

BOUND = 8 * 2.0 ** -23


def bf16(rng, shape, relu=False):
    """Random BF16 bit patterns and their values."""
    u = rng.standard_normal(shape).astype(np.float32)
    if relu:
        u = np.maximum(u, 0.0)
    b = (u.view(np.uint32) + 0x8000 >> 16).astype(np.uint16)
    return b, (b.astype(np.uint32) << 16).view(np.float32).astype(np.float64)


# every layer's channels: first source (up: at half resolution), second, output
LAYERS = [(2, 0, 0, 16), (16, 0, 0, 16), (16, 0, 0, 32), (32, 0, 0, 32), (32, 0, 0, 64), (64, 0, 0, 64),
          (64, 32, 1, 32), (32, 16, 1, 16), (16, 0, 0, 1)]


@pytest.mark.parametrize("X, Y, Z", [(4, 4, 8), (14, 8, 8), (64, 16, 8), (32, 32, 34)])
@pytest.mark.parametrize("c1, c2, up, co", LAYERS)
def test_against_64_bit_sums(gpu, X, Y, Z, c1, c2, up, co):
    rng = np.random.default_rng(X + c1)
    def ptr(a, t):
        return None if a is None else a.ctypes.data_as(C.POINTER(t))
    x32 = h32 = b1 = b2 = bh = None
    if c1 == 2:
        x32 = rng.standard_normal((Z, Y, X, 2)).astype(np.float32)
        x = x32.astype(np.float64)
    else:
        b1, x = bf16(rng, (Z // 2, Y // 2, X // 2, c1) if up else (Z, Y, X, c1), relu=True)
        if up:
            x = x.repeat(2, 0).repeat(2, 1).repeat(2, 2)
        if c2:
            b2, v = bf16(rng, (Z, Y, X, c2), relu=True)
            x = np.concatenate([x, v], axis=-1)
    if co == 1:
        h32 = rng.standard_normal((Z, Y, X, 1)).astype(np.float32)
        h = h32.astype(np.float64)
    else:
        bh, h = bf16(rng, (Z, Y, X, co))
    dw = np.zeros((27, co, c1 + c2), np.float32)
    u16, f32 = C.c_uint16, C.c_float
    assert native.load().picgpu_test_conv3d_dw(X, Y, Z, c1, c2, up, co, ptr(b1, u16), ptr(b2, u16), ptr(bh, u16),
                                               ptr(x32, f32), ptr(h32, f32), ptr(dw, f32)) == abi.OK
    xp = np.zeros((Z + 2, Y + 2, X + 2, c1 + c2))
    xp[1:-1, 1:-1, 1:-1] = x
    hv = h.reshape(-1, co)
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        ref = hv.T @ xp[dz:dz + Z, dy:dy + Y, dx:dx + X].reshape(-1, c1 + c2)
        # against the norm of the sums of magnitudes where the signs cancel
        scale = np.linalg.norm(ref) + 2.0 ** -4 * np.linalg.norm(abs(hv).T @ abs(
            xp[dz:dz + Z, dy:dy + Y, dx:dx + X]).reshape(-1, c1 + c2)) / np.sqrt(len(hv))
        assert np.linalg.norm(dw[t] - ref) <= BOUND * scale, t
