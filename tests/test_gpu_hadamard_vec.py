"""The vector kernels' M2L Hadamard step (k_m2l_had_v64, k_m2l_had_v32): FP64
against the oracle, the mixed form against the FP64 form for every block width
of right-hand sides, with symmetric translation blocks and with tables whose
blocks are not symmetric (replaced through fmmg_operator)."""
import os

import numpy as np
import pytest

import fmmg
import oracle as O
from gpu_common import SEED, gpu_eval, points, rel_l2, share_operators, unit_normals

pytestmark = pytest.mark.gpu


def _skew(lib):
    """Scale every component of every translation by a factor of its own: the
    3 x 3 blocks are no longer symmetric."""
    n_sp = {311: 12, 511: 9}[lib.kt]
    scale = 1.0 + 0.01 * np.arange(n_sp)
    for i in range(316):
        t = lib.operator(4, i).reshape(-1, n_sp, 2)
        lib.set_operator(4, i, t * scale[None, :, None])


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("kt,np_,kind,n", [(311, 4, "sphere_clusters", 6000), (311, 5, "uniform", 700),
                                           (511, 4, "uniform", 5003), (511, 5, "sphere_clusters", 3001)])
def test_vector_hadamard(kt, np_, kind, n, skew):
    """Sparse and full child sets, few and many target parents.  np = 5 leaves
    a ragged last slice of frequencies on the mixed form's grid (405 = 8 x 50 +
    5).  FP64: the 1e-10 parity gate.  Mixed against FP64: FP32 sums through
    the factored pseudo-inverses differ by a few 1e-6 at np <= 5; 2e-5 bounds
    that with the skewed tables' larger cancellation."""
    import torch
    rng = np.random.default_rng(SEED + kt + np_)
    src = points(kind, n, rng)
    lib = fmmg.FMM3d(kt, np_=np_, pts_max=20, coefs=(1.0, 0.3))
    lib.setup(src)
    if skew:
        _skew(lib)
    orc = O.Oracle(kt, np_=np_, pts_max=20, coefs=(1.0, 0.3), nthreads=os.cpu_count() or 1)
    orc.setup(src, src, src)
    share_operators(lib, orc)
    den = rng.uniform(-1, 1, (13, n * 3))
    ref = [gpu_eval(lib, den[r]) for r in range(13)]
    assert rel_l2(ref[0], orc.evaluate(den[0])) <= 1e-10
    for k in (1, 2, 3, 5, 8, 12, 13):  # blocks of 1, 2, 4, 8, 8, 4 x 3 and 8 x 2 right-hand sides
        d = torch.from_numpy(den[:k].copy()).cuda()
        out = torch.zeros(k, n * 3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        lib.evaluate_device(d, out, k, fmmg.PREC_MIXED)
        lib.sync()
        v = out.cpu().numpy()
        worst = max(rel_l2(v[r], ref[r]) for r in range(k))
        print("kernel %d np %d k %d skew %d mixed-vs-fp64 %.2e" % (kt, np_, k, skew, worst))
        assert worst <= 2e-5


def test_vector_adjoint_follows_spectrum_layout():
    """<w, A s> = <A^T w, s> to FP64 rounding for the Stokes and Navier kernels,
    whose transposed step reads and writes the same component-major spectra
    (1e-11: the two sides' sums differ in order through the np = 4 operators)."""
    rng = np.random.default_rng(SEED)
    for kt in (311, 511):
        n = 3000
        src = points("sphere_clusters", n, rng)
        lib = fmmg.FMM3d(kt, np_=4, pts_max=20, coefs=(1.0, 0.3))
        lib.setup(src, unit_normals(rng, n))
        s, w = rng.uniform(-1, 1, n * 3), rng.uniform(-1, 1, n * 3)
        g, _ = lib.adjoint(w)
        a, b = float(w @ gpu_eval(lib, s)), float(g.ravel() @ s)
        assert abs(a - b) <= 1e-11 * np.linalg.norm(w) * np.linalg.norm(gpu_eval(lib, s))
