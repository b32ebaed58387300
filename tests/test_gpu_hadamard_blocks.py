"""Scalar Hadamard step in blocks of 2, 4 and 8 right-hand sides and with few
target parents a CTA, against the FP64 form and between its forms."""
import numpy as np
import pytest

import fmmg
from gpu_common import SEED, gpu_eval, points, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_,n,kind", [(4, 600, "uniform"), (5, 9001, "sphere_clusters"), (6, 20000, "uniform")])
def test_scalar_hadamard_blocks(np_, n, kind):
    """Mixed within 1e-5 of FP64 (2e-6 seen at np <= 6); each right-hand side is
    computed with the same operations in blocks of any width (form 4) and in
    form 3's blocks of 8, so these agree bit for bit."""
    import torch
    rng = np.random.default_rng(SEED + n)
    src = points(kind, n, rng)
    lib = fmmg.FMM3d(111, np_=np_, pts_max=20)
    lib.setup(src)
    den = rng.normal(size=(12, n))
    d = torch.from_numpy(den).cuda()
    ref = np.stack([gpu_eval(lib, den[r]) for r in range(3)])
    for k in (2, 3, 4, 5, 8, 9, 12):
        got = {}
        for form in (4, 3):
            lib.tuning({"had_fp32_rhs_per_thread": form})
            out = torch.zeros(k, n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            lib.evaluate_device(d[:k].contiguous(), out, k, fmmg.PREC_MIXED)
            lib.sync()
            got[form] = out.cpu().numpy()
        assert np.array_equal(got[3], got[4])
        for r in range(min(k, 3)):
            assert rel_l2(got[4][r], ref[r]) <= 1e-5
