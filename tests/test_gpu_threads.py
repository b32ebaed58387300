"""Handles of different orders in use by several threads at once."""
import threading
import time

import numpy as np
import pytest

import fmmg
from gpu_common import SEED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [fmmg.PREC_FP64, fmmg.PREC_MIXED])
@pytest.mark.parametrize("kt", [111, 311])
def test_handles_of_two_orders_at_once(kt, form):
    """Four threads evaluate on handles of np 3, 8, 8 and 8 for two seconds: the
    kernels whose shared memory depends on the order launch for all, with the
    results of each handle alone, bit for bit."""
    rng = np.random.default_rng(SEED)
    n = 400
    x = rng.random((n, 3))
    x[::2] *= 0.05  # a corner refined deeper: W lists
    den = rng.normal(size=n * fmmg.KERNELS[kt][0])
    handles, want = [], []
    for np_ in (3, 8, 8, 8):
        f = fmmg.FMM3d(kt, np_=np_, pts_max=20)
        f.setup(x)
        f.set_precision(form)
        handles.append(f)
        want.append(f.evaluate(den))
    assert handles[0].worklist(1)[0].size > 0
    end = time.time() + 2.0
    errors, calls = [], [0] * 4

    def run(i):
        try:
            while time.time() < end and not errors:
                assert np.array_equal(handles[i].evaluate(den), want[i])
                calls[i] += 1
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert min(calls) > 10
