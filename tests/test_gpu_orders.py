"""V-list DFTs at the smallest order and at the large ones (few grids per block,
long lines).

Bars: the plain form against the oracle 1e-12 (the same operators, as in
test_gpu_parity.py) and against the direct sum about four times the truncation
error of these orders (2.7e-11 at m = 12, 1.2e-13 at m = 16, where FP64
rounding takes over, with 200k uniform points); the mixed form's 1e-6.
"""
import ctypes

import numpy as np
import pytest

import pvfmm_b200 as P
from oracle import pvfmm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 10, 12])
def test_orders_match_oracle(m):
    rng = np.random.default_rng(m)
    x, q = rng.random((2000, 3)), rng.uniform(-1, 1, (2000, 1))
    ops = O.Operators.from_arrays(O.KERNELS[0], m, P.precomp_operators(P.FMMKernel.LaplacePotential, m))
    want = O.pvfmm_eval(0, m, 30, x, q, x, ops=ops)
    ctx = P.FMMParticleContext(-1, 30, m, P.FMMKernel.LaplacePotential)
    out = ctx.evaluate(x.reshape(-1), q.reshape(-1), None, x.reshape(-1), True)
    assert ctx.tree_stats()["n_vtrg"] > 16
    assert O.rel_l2(out.reshape(-1, 1), want) < 1e-12


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


def test_mixed_potentials_at_order_10():
    """The V-list's FP32 rounding shows most at m = 10.  Median relative error
    of the potentials against the plain form, geometric mean over eight point
    sets: 2.05e-7 with chained FP32 sums along x, 2.38e-7 with paired ones
    (higher in each set).  The bar lies between."""
    logs = []
    ctx = [P.FMMParticleContext(-1, 120, 10, P.FMMKernel.LaplacePotential, precision=p)
           for p in (P.PRECISION_MIXED, P.PRECISION_PLAIN)]
    for seed in range(8):
        rng = np.random.default_rng(seed)
        centres = rng.uniform(0.1, 0.9, (8, 3))
        x = np.clip(centres[rng.integers(0, 8, 100_000)] + 0.02 * rng.standard_normal((100_000, 3)), 0, 1).reshape(-1)
        q = rng.uniform(-1, 1, 100_000)
        a, b = (c.evaluate(x, q, None, x, True) for c in ctx)
        logs.append(np.log(np.median(np.abs(a - b) / np.abs(b))))
    assert np.exp(np.mean(logs)) < 2.2e-7
