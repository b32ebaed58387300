"""The mixed form's downward pass through the folded product C2E x L2L, on the
built tables and on a replaced L2L table, over trees of several depths."""
import numpy as np
import pytest

import fmmg
from gpu_common import SEED, gpu_eval, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,np_,n,pts", [(111, 4, 3, 1), (111, 6, 9000, 5), (121, 5, 4000, 30), (311, 4, 3000, 4),
                                          (511, 4, 3000, 20)])
def test_mixed_downward_fold(kt, np_, n, pts):
    """Mixed against FP64 on the same tables, 2e-5 (4e-6 seen at np <= 6: FP32
    sums through the factored pseudo-inverses)."""
    import torch
    rng = np.random.default_rng(SEED + n)
    src = rng.random((n, 3)) * np.where(np.arange(n)[:, None] % 2, 1.0, 0.1)  # a corner refined deeper
    nrm = rng.normal(size=(n, 3))
    lib = fmmg.FMM3d(kt, np_=np_, pts_max=pts, coefs=(1.0, 0.3))
    lib.setup(src, nrm / np.linalg.norm(nrm, axis=1)[:, None])
    den = rng.normal(size=(3, n * lib.sd))
    d = torch.from_numpy(den).cuda()
    out = torch.zeros(3, lib.nt * lib.td, dtype=torch.float64, device="cuda")
    for replaced in (False, True):
        if replaced:
            for o in range(8):
                lib.set_operator(3, o, lib.operator(3, o) * (0.5 + 0.1 * o))
        ref = [gpu_eval(lib, den[r]) for r in range(3)]
        torch.cuda.synchronize()
        lib.evaluate_device(d, out, 3, fmmg.PREC_MIXED)
        lib.sync()
        v = out.cpu().numpy()
        for r in range(3):
            assert rel_l2(v[r], ref[r]) <= 2e-5
