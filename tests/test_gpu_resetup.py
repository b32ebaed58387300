"""Handles that are set up again: after a setup that ran out of device memory,
with and without replaced operator tables, and what they keep of the device's
memory."""
import contextlib

import numpy as np
import pytest

import fmmg
from gpu_common import SEED, rel_l2

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def _little_memory(leave):
    """About `leave` bytes of the device's memory free."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = [torch.empty(max(free - leave, 1), dtype=torch.uint8, device="cuda")]
    try:
        yield
    finally:
        hold.clear()
        torch.cuda.empty_cache()


def _fail_setup(f, rng):
    """A setup of f that runs out of device memory while the plan is built."""
    big = rng.random((8000000, 3))  # 192 MB of coordinates
    with _little_memory(48 * MB), pytest.raises(fmmg.FmmgError):
        f.setup(big)


def test_setup_after_a_setup_out_of_memory():
    """The failed allocation is reported once: the next setup of the handle works."""
    rng = np.random.default_rng(SEED)
    f = fmmg.FMM3d(111, np_=4, pts_max=40)
    x, den = rng.random((3000, 3)), rng.normal(size=3000)
    f.setup(x)
    want = f.evaluate(den)
    _fail_setup(f, rng)
    f.setup(x)
    assert np.array_equal(f.evaluate(den), want)
