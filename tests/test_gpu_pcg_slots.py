"""Calls of different sizes in turn through the allocation-free PCG entry point:
the values that its blocks exchange lie in one scratch array, and what an
earlier call of another size left there must not pass for this call's.  A size
gives the same bits each time, and they solve the system."""
import ctypes as C

import numpy as np
import pytest

from picfoam_gb300 import abi, native
from test_zz_no_alloc import laplacian_ell

pytestmark = pytest.mark.gpu


def test_sizes_in_turn(gpu):
    torch = pytest.importorskip("torch")
    lib = native.load()
    tol, first = 1e-10, {}
    for n in (10, 30, 6, 30, 16, 10, 40, 16, 6, 40):
        diag, off, nbr, _ = laplacian_ell(n, 0.004)
        b = np.random.default_rng(n).standard_normal(n ** 3)
        d = [torch.tensor(v, device="cuda") for v in (diag, off, nbr, b, np.zeros(n ** 3))]
        iters, res = C.c_int(-1), C.c_double(-1.0)
        status = lib.picgpu_solve_ldu_noalloc(n ** 3, *[v.data_ptr() for v in d], tol, 20000, C.byref(iters),
                                              C.byref(res), None)
        assert status == abi.OK and 0 < iters.value and res.value <= tol
        x = d[4].cpu().numpy()
        near = nbr.reshape(-1, 6)
        mx = diag * x + (off.reshape(-1, 6) * np.where(near >= 0, x[np.maximum(near, 0)], 0.0)).sum(axis=1)
        # the true residual: the recursive one and its drift, of the order of
        # iterations x 2^-53 x |M| |x| / |b|, far below tol here
        assert np.linalg.norm(b - mx) <= 2.0 * tol * np.linalg.norm(b)
        x0, k0 = first.setdefault(n, (x, iters.value))
        assert np.array_equal(x, x0) and iters.value == k0
