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


def _outputs(f, den, w):
    """FP64, mixed (2 right-hand sides) and transposed results of f."""
    import torch
    d = torch.from_numpy(den).cuda()
    out = torch.zeros(2, f.nt * f.td, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f.evaluate_device(d, out, 2, fmmg.PREC_MIXED)
    f.sync()
    return {"fp64": f.evaluate(den[0]), "mixed": out.cpu().numpy(), "adjoint": f.adjoint(w)[0]}


def _inputs(kt, n, rng):
    x, den = rng.random((n, 3)), rng.normal(size=(2, n * fmmg.KERNELS[kt][0]))
    return x, den, rng.normal(size=n * fmmg.KERNELS[kt][1])


# both forms of a handle run the same kernels on the same tables, so the
# results are the same bit for bit but for the mixed form's split-K sums, which
# run in one order too
@pytest.mark.parametrize("kt", [111, 311])
@pytest.mark.parametrize("when", ["evaluated", "not evaluated"])
def test_replaced_table_after_a_failed_setup(kt, when):
    """A table replaced between a setup that failed and the next one is the one
    that the next setup's evaluates use, as on a fresh handle."""
    rng = np.random.default_rng(SEED + kt)
    x, den, w = _inputs(kt, 3000, rng)
    f = fmmg.FMM3d(kt, np_=4, pts_max=40)
    f.setup(x)
    if when == "evaluated":
        _outputs(f, den, w)
    _fail_setup(f, rng)
    g = fmmg.FMM3d(kt, np_=4, pts_max=40)
    for h in (f, g):
        h.set_operator(2, 0, h.operator(2, 0) * 1.5)
        for i in range(0, 316, 5):
            h.set_operator(4, i, h.operator(4, i) * 0.75)
        h.setup(x)
    got, want = _outputs(f, den, w), _outputs(g, den, w)
    for key in want:
        assert np.array_equal(got[key], want[key]), key


@pytest.mark.parametrize("kt,form", [(111, fmmg.PREC_FP64), (311, fmmg.PREC_FP64), (311, fmmg.PREC_MIXED)])
def test_replaced_table_waits_for_queued_evaluates(kt, form):
    """evaluate_device only queues work: tables replaced right after it serve the
    calls that follow and not the ones that still run (several milliseconds of
    them), down to the last bit."""
    import torch
    rng = np.random.default_rng(SEED)
    n, calls = 100000, 6
    st = torch.cuda.Stream()
    f = fmmg.FMM3d(kt, np_=4, pts_max=40, stream=st.cuda_stream)
    f.setup(rng.random((n, 3)))
    den = torch.from_numpy(rng.normal(size=n * f.sd)).cuda()
    out = torch.zeros(calls + 1, n * f.td, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tables = [f.operator(4, i) for i in range(0, 316, 7)]
    values = {}
    for scale in (1.0, 0.5):
        for j, i in enumerate(range(0, 316, 7)):
            f.set_operator(4, i, tables[j] * scale)
        f.evaluate_device(den, out[0], 1, form)
        f.sync()
        values[scale] = out[0].cpu().numpy()
    now = 0.5
    for scale in (1.0, 0.5, 1.0):
        for c in range(calls):
            f.evaluate_device(den, out[c], 1, form)
        for j, i in enumerate(range(0, 316, 7)):
            f.set_operator(4, i, tables[j] * scale)
        f.evaluate_device(den, out[calls], 1, form)
        f.sync()
        got = out.cpu().numpy()
        for c in range(calls):
            assert np.array_equal(got[c], values[now])
        assert np.array_equal(got[calls], values[scale])
        now = scale


def test_mixed_staging_is_given_back():
    """What a handle's first mixed call stages on the device (some 300 MB of FP64
    operators for Navier at np = 8) does not stay with the process."""
    import torch
    rng = np.random.default_rng(SEED)
    x, den, w = _inputs(511, 500, rng)

    def free_after(mixed):
        f = fmmg.FMM3d(511, np_=8, pts_max=40, coefs=(1.0, 0.3))
        f.setup(x)
        f.evaluate(den[0])
        if mixed:
            _outputs(f, den, w)
        f.close()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    free_after(False)
    before = free_after(False)
    free_after(True)  # the kernels' code
    assert free_after(True) >= before - 64 * MB


@pytest.mark.parametrize("kt", [111, 311])
def test_mixed_call_after_mixed_calls_out_of_memory(kt):
    """First mixed calls that run out of device memory at any of their
    allocations are refused, and the next call of the handle with the memory
    back is the fresh handle's."""
    rng = np.random.default_rng(SEED + kt)
    x, den, w = _inputs(kt, 2000, rng)
    x[::2] *= 0.1  # a corner refined deeper: W lists
    g = fmmg.FMM3d(kt, np_=6, pts_max=40)
    g.setup(x)
    want = _outputs(g, den, w)
    refused = 0
    f = fmmg.FMM3d(kt, np_=6, pts_max=40)
    f.setup(x)
    f.set_precision(fmmg.PREC_MIXED)
    for leave in list(range(2, 40, 6)) + list(range(40, 200, 20)):
        with _little_memory(leave * MB):
            try:
                assert rel_l2(f.evaluate(den[0]), want["mixed"][0]) <= 1e-5
            except fmmg.FmmgError:
                refused += 1
        if leave % 4 == 0:  # a new setup keeps the operator tables' blocks that were allocated
            f.setup(x)
    assert refused >= 3
    f.set_precision(fmmg.PREC_FP64)
    got = _outputs(f, den, w)
    for key in want:
        assert np.array_equal(got[key], want[key]), key


def test_setup_out_of_host_memory_leaves_the_handle_as_it_was():
    """A new setup that cannot hold the built tables again (host memory) is
    refused before it gives up anything: the handle still evaluates, on its
    replaced tables, and the next setup works."""
    import resource
    rng = np.random.default_rng(SEED)
    x, den, w = _inputs(311, 2000, rng)
    f = fmmg.FMM3d(311, np_=6, pts_max=40)
    f.setup(x)
    built = f.evaluate(den[0])
    f.set_operator(3, 2, f.operator(3, 2) * 1.5)
    want = _outputs(f, den, w)
    old = resource.getrlimit(resource.RLIMIT_AS)
    resource.setrlimit(resource.RLIMIT_AS, (1 << 20, old[1]))  # no further mappings: the tables take 46 MB
    try:
        with pytest.raises(fmmg.FmmgError) as e:
            f.setup(x)
    finally:
        resource.setrlimit(resource.RLIMIT_AS, old)
    assert e.value.status == fmmg.FMMG_OOM
    got = _outputs(f, den, w)
    for key in want:
        assert np.array_equal(got[key], want[key]), key
    f.setup(x)
    assert np.array_equal(f.evaluate(den[0]), built)


def test_translation_layouts_change_in_place():
    """Tables replaced back and forth between symmetric and general 3 x 3 blocks
    take no more device memory each time (77 and 112 MB in FP64 at np = 7) than
    the first."""
    import torch
    rng = np.random.default_rng(SEED)
    x, den, w = _inputs(311, 500, rng)
    f = fmmg.FMM3d(311, np_=7, pts_max=40)
    f.setup(x)
    table = f.operator(4, 0)
    general = (table.reshape(-1, 12, 2) * np.linspace(1.0, 1.1, 12)[None, :, None]).ravel()
    free = []
    for _ in range(4):
        for t in (general, table):
            f.set_operator(4, 0, t)
            _outputs(f, den, w)
        torch.cuda.empty_cache()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[-1] >= free[0] - 16 * MB


@pytest.mark.parametrize("kt", [111, 311])
def test_replaced_tables_go_with_the_next_setup(kt):
    """Replaced tables (for 311 with 3 x 3 blocks that are not symmetric) serve
    the evaluates until the next setup, which goes back to the built ones in
    every form, and keeps those through further setups."""
    rng = np.random.default_rng(SEED + kt)
    x, den, w = _inputs(kt, 3000, rng)
    y = rng.random((2500, 3))
    den_y, w_y = den[:, :2500 * fmmg.KERNELS[kt][0]].copy(), w[:2500 * fmmg.KERNELS[kt][1]].copy()
    g = fmmg.FMM3d(kt, np_=4, pts_max=40)
    g.setup(x)
    want = _outputs(g, den, w)
    f = fmmg.FMM3d(kt, np_=4, pts_max=40)
    f.setup(x)
    first = _outputs(f, den, w)
    n_sp = 12 if kt == 311 else 1
    scale = np.linspace(1.0, 1.1, n_sp)
    for i in range(316):
        f.set_operator(4, i, f.operator(4, i).reshape(-1, n_sp, 2) * scale[None, :, None])
    f.set_operator(3, 2, f.operator(3, 2) * 1.5)
    replaced = _outputs(f, den, w)
    for key in want:
        assert np.array_equal(first[key], want[key]), key
        assert rel_l2(replaced[key], want[key]) > 1e-3, key  # the replaced tables are in use
    f.setup(y)
    g2 = fmmg.FMM3d(kt, np_=4, pts_max=40)
    g2.setup(y)
    got, ref = _outputs(f, den_y, w_y), _outputs(g2, den_y, w_y)
    f.setup(x)
    again = _outputs(f, den, w)
    for key in want:
        assert np.array_equal(got[key], ref[key]), key
        assert np.array_equal(again[key], want[key]), key
