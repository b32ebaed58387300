"""Near-field kernels at the edges of their target blocks: leaves of 1 to several
blocks of targets (a leaf at the depth limit holds any number), few leaves and
many, targets apart from the sources, one to 9 right-hand sides."""
import numpy as np
import pytest

import fmmg
from gpu_common import SEED, gpu_eval, rel_l2, unit_normals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", [111, 121, 312, 321, 511, 521])
@pytest.mark.parametrize("n,n_trg,pts,levels", [(1, 1, 1, 30), (200, 331, 300, 30), (3001, 64, 3001, 1),
                                                (900, 8300, 40, 2), (17000, 0, 2, 30)])
def test_near_field_blocks(kt, n, n_trg, pts, levels):
    """U-list sums alone against the dense sum of the whole evaluate where one
    leaf holds everything (no far field), else FP64 against the mixed form;
    FP64 1e-12 (sums of the same terms in another order), mixed 2e-6 (FP32 sums
    of at most 128 terms) with 2e-5 for the kernels with cancelling normals."""
    import torch
    rng = np.random.default_rng(SEED + n + kt)
    src, nrm = rng.random((n, 3)), unit_normals(rng, n)
    trg = rng.random((n_trg, 3)) if n_trg else src
    lib = fmmg.FMM3d(kt, np_=3, pts_max=pts, max_level=levels, coefs=(1.0, 0.3))
    lib.setup(src, nrm, trg)
    k = 9
    den = rng.normal(size=(k, n * lib.sd))
    d = torch.from_numpy(den).cuda()
    ref = np.stack([gpu_eval(lib, den[r], fmmg.STAGE_U) for r in range(k)])
    if lib.info()["max_depth"] <= 1:  # everything is near
        _, _, dense = lib.check(den[0], gpu_eval(lib, den[0]), np.arange(lib.nt))
        assert rel_l2(ref[0], dense) <= 1e-12
    out = torch.zeros(lib.nt * lib.td, dtype=torch.float64, device="cuda")
    tol = 2e-5 if kt in (121, 321, 521) else 2e-6
    for r in range(2):
        torch.cuda.synchronize()
        lib.evaluate_stages(d[r], out, fmmg.STAGE_U, fmmg.PREC_MIXED)
        lib.sync()
        assert rel_l2(out.cpu().numpy(), ref[r]) <= tol
    full = torch.zeros(k, lib.nt * lib.td, dtype=torch.float64, device="cuda")
    one = torch.zeros(k, lib.nt * lib.td, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for r in range(k):
        lib.evaluate_device(d[r].contiguous(), one[r], 1, fmmg.PREC_MIXED)
    lib.sync()
    want = one.cpu().numpy()
    for kk in (2, 3, 4, 8, 9):  # blocks of 2, 2 + 1, 4, 8, 8 + 1 (vector kernels 2, 2 + 1, 4, 4 + 4, 4 + 4 + 1)
        full.zero_()
        torch.cuda.synchronize()
        lib.evaluate_device(d[:kk].contiguous(), full, kk, fmmg.PREC_MIXED)
        lib.sync()
        got = full.cpu().numpy()
        for r in range(kk):  # every right-hand side of every block
            assert rel_l2(got[r], want[r]) <= 2e-5


@pytest.mark.parametrize("kt", [111, 121, 311])
@pytest.mark.parametrize("pts", [2, 9, 12])
def test_near_field_of_small_leaves(kt, pts):
    """Trees on either side of the points a leaf below which one warp takes it
    (near_f64.cuh), with more than 16 leaves an SM: the evaluate against dense
    sums at some targets (np = 6 truncates at 1e-6 to 1e-5; a near pair missed
    or counted twice is 1e-2 here), the transposed sums through <w, A s> =
    <A^T w, s>, and the target gradient against dense sums."""
    rng = np.random.default_rng(SEED + kt + pts)
    n = 9000 if pts < 5 else 60000
    src, nrm = rng.random((n, 3)), unit_normals(rng, n)
    lib = fmmg.FMM3d(kt, np_=6, pts_max=pts)
    lib.setup(src, nrm)
    assert len(lib.worklist(0)[0]) > 16 * 148
    s, w = rng.uniform(-1, 1, n * lib.sd), rng.uniform(-1, 1, n * lib.td)
    v = gpu_eval(lib, s)
    idx = rng.choice(n, 300, replace=False)
    rel, _, _ = lib.check(s, v, idx)
    assert rel <= 1e-4
    g, _ = lib.adjoint(w)
    assert abs(float(w @ v) - float(g.ravel() @ s)) <= 1e-11 * np.linalg.norm(w) * np.linalg.norm(v)
    if kt == 111:  # d/dx of w(x) sum_y den(y) / (4 pi |x - y|)
        _, grad = lib.adjoint(w, s, target_grad=True)
        d = src[idx, None, :] - src[None, :, :]
        r = np.sqrt((d * d).sum(-1))
        r[r == 0] = np.inf
        dense = -(w[idx, None] / (4 * np.pi)) * (d * (s[None, :] / r**3)[..., None]).sum(1)
        assert rel_l2(grad[idx], dense) <= 1e-4
