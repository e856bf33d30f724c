"""FP64 products of translate.cu at the edges of their dispatch: the choice of
the row tile, and the parent-child products that leave out empty children.

Bar: sums of K products of N(0,1) values in FP64, 1e-14 of the largest value
per 64 terms (as in test_gpu_reference.py).
"""
import ctypes

import numpy as np
import pytest

import pvfmm_b200 as P

pytestmark = pytest.mark.gpu

VP = ctypes.c_void_p


def _p(a):
    return None if a is None else a.ctypes.data_as(VP)


# 296 blocks of 128 x 64 take the 32-row tiles, more the 128-row ones; rows and
# columns beyond and below whole tiles; K below, at and beyond whole steps
@pytest.mark.parametrize("M,N,K", [(1, 8, 2), (31, 56, 16), (33, 66, 18), (128 * 296, 64, 20),
                                   (128 * 296 + 1, 64, 20), (9001, 296, 296), (12800, 152, 34)])
def test_row_tiles(M, N, K):
    f = P.load_library().PVFMMB200TranslateGemmCheck
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_long, ctypes.c_int, ctypes.c_int, VP, ctypes.c_long, VP, VP, VP, ctypes.c_long, VP, VP,
                  ctypes.c_int, ctypes.c_int]
    rng = np.random.default_rng(M + N + K)
    A, B, C = rng.standard_normal((M, K)), rng.standard_normal((K, N)), np.zeros((M, N))
    assert f(M, N, K, _p(A), M, None, _p(B), _p(C), M, None, None, 0, 1) == 0, P.last_error()
    want = A @ B
    assert np.abs(C - want).max() < 1e-14 * max(1, K / 64) * np.abs(want).max()


# one parent; parents without children, an octant without parents; 32-row tiles
# (up to 296 blocks of 128 x 64 over the 8 octants) and 128-row ones (6000)
@pytest.mark.parametrize("M,dim,keep", [(1, 8, 1.0), (37, 56, 0.4), (129, 56, 0.0), (700, 152, 0.3),
                                        (6000, 56, 0.45)])
def test_children_with_points_only(M, dim, keep):
    f = P.load_library().PVFMMB200ChildProductsCheck
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_long, ctypes.c_int] + [VP] * 7
    rng = np.random.default_rng(M + dim)
    bits = rng.random((M, 8)) < keep
    bits[:, 3] = False
    mask = np.packbits(bits, axis=1, bitorder="little").reshape(-1)
    ch, B, D = (rng.standard_normal(s) for s in ((M, 8, dim), (8, dim, dim), (dim, 8, dim)))
    up_in, down = rng.standard_normal((M, dim)), rng.standard_normal((M, 8, dim))
    up, got = np.full((M, dim), 7.0), down.copy()
    assert f(M, dim, _p(mask), _p(ch), _p(B), _p(up), _p(up_in), _p(D), _p(got)) == 0, P.last_error()
    want = np.einsum("kz,kzi,zij->kj", bits.astype(float), ch, B, optimize=True)
    want_down = down + bits[:, :, None] * np.einsum("ki,izj->kzj", up_in, D, optimize=True)
    scale = 1e-14 * max(1, 8 * dim / 64)
    assert np.abs(up - want).max() <= scale * max(np.abs(want).max(), 1)
    assert np.abs(got - want_down).max() <= scale * np.abs(want_down).max()
    assert np.array_equal(got[~bits], down[~bits])


# trees with enough internal nodes and empty leaves to take the lists, against
# the direct sum; a left-out child would cost 1e-2 and more, the bars are about
# three times the truncation error at m = 6
@pytest.mark.parametrize("kernel,prec,bar", [(P.FMMKernel.LaplacePotential, P.PRECISION_PLAIN, 2e-5),
                                             (P.FMMKernel.StokesVelocity, P.PRECISION_MIXED, 1e-3)])
def test_sparse_tree_matches_direct_sum(kernel, prec, bar):
    rng = np.random.default_rng(17)
    n = 60_000
    u = rng.standard_normal((n, 3))
    x = (0.5 + 0.4 * u / np.linalg.norm(u, axis=1)[:, None]).reshape(-1)
    q = rng.standard_normal(n * P.KERNEL_DIMS[kernel][0])
    ctx = P.FMMParticleContext(-1, 10, 6, kernel, precision=prec)
    out = ctx.evaluate(x, q, None, x, True)
    st = ctx.tree_stats()
    assert st["n_nodes"] - st["n_leaves"] >= 4096 and st["n_tleaf"] < 0.6 * st["n_leaves"]
    k1 = P.KERNEL_DIMS[kernel][1]
    idx = rng.choice(n, 500, replace=False)
    want = P.kernel_eval(kernel, x, q, x.reshape(-1, 3)[idx].reshape(-1).copy()).reshape(-1, k1)
    got = out.reshape(-1, k1)[idx]
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < bar
