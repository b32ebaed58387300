"""The FP64 row GEMM (k_gemm_f64) through the evaluate: trees whose leaf counts
fall on either side of each tile size of launch_gemm_f64, with row scales of 1, 3
and 4 components and several levels in the one launch of the leaves."""
import os
from fractions import Fraction

import numpy as np
import pytest

import fmmg
import oracle as O
from gpu_common import SEED, gpu_eval, rel_l2, share_operators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,np_,n,pts", [(111, 4, 1, 1), (111, 4, 9, 1), (111, 3, 700, 2), (111, 4, 4000, 1),
                                          (111, 4, 9000, 1), (111, 3, 16000, 1), (511, 3, 3000, 1),
                                          (311, 4, 2500, 1), (311, 3, 40, 3)])
def test_fp64_gemm_tiles(kt, np_, n, pts):
    """1e-10 against the oracle's sequential sums on the same operators (4e-13
    seen, from other stages; the order of the products' sums is
    test_fp64_gemm_sums_in_order's)."""
    rng = np.random.default_rng(SEED + n)
    # half of the points in one corner: leaves of several depths
    src = rng.random((n, 3)) * np.where(np.arange(n)[:, None] % 2, 1.0, 0.2)
    lib = fmmg.FMM3d(kt, np_=np_, pts_max=pts, coefs=(1.0, 0.3))
    lib.setup(src)
    orc = O.Oracle(kt, np_=np_, pts_max=pts, coefs=(1.0, 0.3), nthreads=os.cpu_count() or 1)
    orc.setup(src, src, src)
    share_operators(lib, orc)
    den = rng.uniform(-1, 1, n * lib.sd)
    g, c = gpu_eval(lib, den), orc.evaluate(den)
    print("kernel %d np %d: %d leaves, rel_l2 %.1e" % (kt, np_, lib.info()["leaves"], rel_l2(g, c)))
    assert np.linalg.norm(g - c) <= 1e-10 * max(np.linalg.norm(c), 1e-300)


def _fma_chain(x, w):
    """sum over k of w[k] x[k], one correctly rounded multiply-add after another
    from +0 (float() of a fraction rounds to nearest even)."""
    s = 0.0
    for a, b in zip(x, w):
        s = float(Fraction(a) * Fraction(b) + Fraction(s))
    return s


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("K,N,rows,mod", [(2, 1, 1, 1), (14, 9, 17, 3), (16, 16, 16, 4), (18, 81, 3, 1), (50, 33, 5, 3),
                                          (130, 7, 19, 4), (152, 5, 65, 1), (46, 2, 129, 3)])
def test_fp64_gemm_sums_in_order(tile, K, N, rows, mod):
    """Each output is the chain of multiply-adds in ascending k, bit for bit, for
    every tile: values over 12 binary orders of both signs (another order or
    grouping rounds half of the outputs differently), at the edges of the tiles
    (16 values of K a stage, 16 to 128 rows, 16 to 80 outputs)."""
    rng = np.random.default_rng(SEED + 1000 * K + N)
    x = rng.normal(size=(rows, K)) * np.exp2(rng.integers(-6, 7, (rows, K)))
    w = rng.normal(size=(N, K)) * np.exp2(rng.integers(-6, 7, (N, K)))
    sc = np.exp2(rng.integers(-3, 4, mod).astype(float))
    y = np.empty((rows, N))
    st = fmmg.lib().fmmg_selftest_gemm(0, tile, rows, K, N, fmmg._d(x), fmmg._d(w), fmmg._d(sc), mod, fmmg._d(y))
    assert st == fmmg.FMMG_OK
    xs = x * sc[np.arange(K) % mod]
    for r in {0, rows // 2, rows - 1}:
        for n in {0, N // 2, N - 1}:
            assert y[r, n] == _fma_chain(xs[r].tolist(), w[n].tolist())
    assert np.allclose(y, xs @ w.T, rtol=0, atol=1e-12 * np.abs(xs).max() * np.abs(w).max() * K)
