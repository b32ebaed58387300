"""The FP64 row GEMM (k_gemm_f64) through the evaluate: trees whose leaf counts
fall on either side of each tile size of launch_gemm_f64, with row scales of 1, 3
and 4 components and several levels in the one launch of the leaves."""
import os

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
    """1e-10 against the oracle's sequential sums on the same operators: the
    matrix instruction adds in the same order (4e-13 seen, from other stages)."""
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
