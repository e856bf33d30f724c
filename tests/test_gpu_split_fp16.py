"""The mixed form's split-FP16 V-list products (eval.cu, hadamard_tc_kernel
and hadamard_tc3_kernel): scales, empty parents and partial tiles.

Bars: the mixed form's 1e-6 against the plain form for scalar kernels; the
vector kernels also cut the downward pseudo-inverse at FP32 level, so they are
compared with the mixed form's own FP32 SIMT products (1e-6, the bar of that
comparison in test_gpu_parity.py).  Powers of two scale every stored half, sum
and output exactly, so scaled densities give bit-identical scaled outputs.
"""
import numpy as np
import pytest

import pvfmm_b200 as P

pytestmark = pytest.mark.gpu

KERNELS = [(P.FMMKernel.LaplacePotGrad, 8), (P.FMMKernel.StokesPressure, 4), (P.FMMKernel.StokesVelocity, 4)]


def _ctx(kernel, m, precision=P.PRECISION_MIXED, leaf=30):
    return P.FMMParticleContext(-1, leaf, m, kernel, precision=precision)


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _compare(monkeypatch, kernel, m, x, q):
    """The mixed form's outputs and what they are held against."""
    a = _ctx(kernel, m).evaluate(x, q, None, x, True)
    if P.KERNEL_DIMS[kernel][0] == 1:
        return a, _ctx(kernel, m, P.PRECISION_PLAIN).evaluate(x, q, None, x, True)
    monkeypatch.setenv("PVFMM_B200_HADAMARD3", "simt")
    return a, _ctx(kernel, m).evaluate(x, q, None, x, True)


@pytest.mark.parametrize("kernel,m", KERNELS)
@pytest.mark.parametrize("k", [-70, 70])
def test_power_of_two_densities_scale_the_output_exactly(kernel, m, k):
    rng = np.random.default_rng(5)
    x = rng.random(3 * 3001)
    q = rng.standard_normal(3001 * P.KERNEL_DIMS[kernel][0])
    ctx = _ctx(kernel, m)
    a = ctx.evaluate(x, q, None, x, True)
    b = ctx.evaluate(x, np.ldexp(q, k), None, x, False)
    assert np.array_equal(b, np.ldexp(a, k))


# Densities up to where the near field's q/r itself leaves the FP32 range, and
# down to where the smallest output spectra do: the scales of the stored halves
# must not overflow or vanish before that.
@pytest.mark.parametrize("kernel,m", [(P.FMMKernel.LaplacePotential, 8), (P.FMMKernel.StokesVelocity, 4)])
@pytest.mark.parametrize("k", [-90, 112])
def test_whole_fp32_range_of_densities(kernel, m, k):
    rng = np.random.default_rng(6)
    x = rng.random(3 * 3001)
    q = rng.uniform(0.5, 1.0, 3001 * P.KERNEL_DIMS[kernel][0])
    ctx = _ctx(kernel, m)
    a = ctx.evaluate(x, q, None, x, True)
    b = ctx.evaluate(x, np.ldexp(q, k), None, x, False)
    assert np.array_equal(b, np.ldexp(a, k))


# Densities that FP32 rounds to zero (Gaussian weights far out: 1e-306, and
# subnormal FP64 numbers) beside ordinary ones, and alone: 2^-E of such a
# parent has no finite value.
@pytest.mark.parametrize("kernel,m", KERNELS)
@pytest.mark.parametrize("alone", [False, True])
def test_densities_below_the_fp32_range(monkeypatch, kernel, m, alone):
    rng = np.random.default_rng(8)
    pos = rng.random((3001, 3))
    q = rng.standard_normal((3001, P.KERNEL_DIMS[kernel][0]))
    q[pos[:, 0] < 0.5] *= 1e-306
    q[pos[:, 0] < 0.25] *= 1e-14
    x = pos.reshape(-1)
    if alone:
        q[pos[:, 0] >= 0.5] = 0.0
        assert np.all(np.abs(_ctx(kernel, m).evaluate(x, q.reshape(-1), None, x, True)) < 1e-290)
        return
    a, b = _compare(monkeypatch, kernel, m, x, q.reshape(-1))
    assert _rel(a, b) < 1e-6


# 600 / 1500 / 5001 points: 1 V-list target parent below a full tile of 16,
# a few tiles, several tiles per warp with a remainder
@pytest.mark.parametrize("kernel,m", KERNELS)
@pytest.mark.parametrize("n", [600, 1500, 5001])
def test_empty_parents_and_partial_tiles(monkeypatch, kernel, m, n):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3))
    q = rng.standard_normal((n, P.KERNEL_DIMS[kernel][0]))
    # neighbouring parents with exponents of their own: 2^-6 .. 2^6 per cell of
    # side 1/8, so that a parent left out or scaled by another's exponent costs
    # 1e-4 of the result and more
    cell = (pos * 8).astype(int)
    q *= 2.0 ** rng.integers(-6, 7, 512)[cell[:, 0] * 64 + cell[:, 1] * 8 + cell[:, 2]][:, None]
    q[pos[:, 0] < 0.25] = 0.0                       # parents whose spectra are all zero
    a, b = _compare(monkeypatch, kernel, m, pos.reshape(-1), q.reshape(-1))
    assert _rel(a, b) < 1e-6
