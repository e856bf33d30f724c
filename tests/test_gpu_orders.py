"""V-list DFTs at the orders above 10 (one grid per block, long lines).

Bars: the plain form against the direct sum, about four times the truncation
error of these orders (2.7e-11 at m = 12, 1.2e-13 at m = 16, where FP64
rounding takes over, with 200k uniform points); the mixed form's 1e-6.
"""
import ctypes

import numpy as np
import pytest

import pvfmm_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,bar", [(12, 1e-10), (16, 1e-12)])
def test_high_orders_match_direct_sum(monkeypatch, tmp_path, m, bar):
    monkeypatch.setenv("PVFMM_DIR", str(tmp_path))  # the second form reads the first one's factors
    rng = np.random.default_rng(m)
    n = 20_000
    x = rng.random(3 * n)
    q = rng.uniform(-1, 1, n)
    idx = rng.choice(n, 500, replace=False)
    want = P.kernel_eval(P.FMMKernel.LaplacePotential, x, q, x.reshape(-1, 3)[idx].reshape(-1).copy()).reshape(-1)
    for prec, tol in ((P.PRECISION_PLAIN, bar), (P.PRECISION_MIXED, 1e-6)):
        ctx = P.FMMParticleContext(-1, 60, m, P.FMMKernel.LaplacePotential, precision=prec)
        out = ctx.evaluate(x, q, None, x, True)
        assert ctx.tree_stats()["n_vtrg"] > 16
        ctx.close()
        assert np.linalg.norm(out[idx] - want) / np.linalg.norm(want) < tol


@pytest.mark.parametrize("prec", [P.PRECISION_PLAIN, P.PRECISION_MIXED])
@pytest.mark.parametrize("m", [6, 8, 12, 14, 16])
def test_dft_lines_stay_in_registers(prec, m):
    """A thread of the DFT kernels holds its whole line; a launch bound for
    more threads than the order's blocks have would spill it."""
    f = P.load_library().PVFMMB200DftLocalBytes
    up, dn = ctypes.c_int(-1), ctypes.c_int(-1)
    assert f(int(prec), m, ctypes.byref(up), ctypes.byref(dn)) == 0, P.last_error()
    assert (up.value, dn.value) == (0, 0)
