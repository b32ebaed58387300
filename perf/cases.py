"""The evaluator's workloads as timed cases: calls that a program using this
framework makes, through its public Python entry points (fmmg.FMM3d,
fmmg_torch.fmm_apply, droplets.FmmVelocity), from a few thousand points to the
million-point benchmark workload.

A case names the kernel, the surface order np, the leaf size, the point set,
the numbers of points and right-hand sides, the arithmetic ("fp64", the plain
form, or "mixed") and the call:
  device  evaluate_device on CUDA tensors, on the program's torch stream (a
          solver that applies the operator between its own torch operations);
  graph   the same with set_graph(True), as a program that applies one
          operator many times on fixed buffers runs it;
  host    evaluate() on numpy arrays, the drop-in for FMM3d_MPI::evaluate;
  grad    fmmg_torch.fmm_apply forward and backward, gradients with respect to
          the densities and the target positions;
  moving  droplets.FmmVelocity: setup and evaluate at positions that change
          with every call, as a time stepper does.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmm-g_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import droplets  # noqa: E402
import fmmg  # noqa: E402
import fmmg_torch  # noqa: E402
import workloads  # noqa: E402

NORMALS = (121, 321, 322, 521)  # the double-layer kernels


def _case(name, kernel, np_, pts_max, points, n, k, precision, call, n_trg=0, nu=0.25):
    c = dict(kernel=kernel, np=np_, pts_max=pts_max, points=points, n=n, n_trg=n_trg, k=k, precision=precision,
             call=call, nu=nu)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a few thousand points, where launches and the
        # chain of tree levels are the time (the size of the smoke check)
        _case("laplace_4k", 111, 4, 40, "uniform", 4000, 1, "fp64", "device"),
        # the reference driver's own use, evaluate() on host arrays in FP64
        # (low-accuracy configuration: np 4, 150 points a leaf)
        _case("laplace_64k_host", 111, 4, 150, "uniform", 65536, 1, "fp64", "host"),
        # one right-hand side in the mixed form, as an iterative solver asks
        _case("laplace_100k_mixed", 111, 6, 64, "sphere_clusters", 100000, 1, "mixed", "device"),
        # a boundary double layer evaluated at fewer targets off the sources;
        # odd order, odd sizes, three right-hand sides
        _case("laplace_dl_50k_apart", 121, 5, 60, "sphere", 50021, 3, "mixed", "device", n_trg=30011),
        # the benchmark workload in both forms, replayed as a CUDA graph
        _case("laplace_1m_fp64", 111, 6, 64, "sphere_clusters", 1 << 20, 1, "fp64", "graph"),
        _case("laplace_1m_mixed_k8", 111, 6, 64, "sphere_clusters", 1 << 20, 8, "mixed", "graph"),
        # more right-hand sides than a launch block holds, and a ragged rest
        _case("laplace_250k_np7_k13", 111, 7, 100, "uniform", 250007, 13, "mixed", "device"),
        # training through the operator: value, density and position gradients
        _case("laplace_grad_128k", 111, 6, 64, "uniform", 131072, 2, "fp64", "grad"),
        # Stokes double layer on many bodies, 8 right-hand sides
        _case("stokes_dl_150k_k8", 321, 6, 64, "ellipsoids", 150000, 8, "mixed", "device"),
        # Stokes single layer on the same bodies in FP64, one right-hand side
        _case("stokes_sl_60k_fp64", 311, 6, 64, "ellipsoids", 60007, 1, "fp64", "device"),
        # elasticity at high accuracy
        _case("navier_120k_np8_k4", 511, 8, 64, "shell", 120000, 4, "mixed", "device", nu=0.3),
        # sedimenting droplets: the points move, so every pass sets up again
        _case("droplets_30k", 311, 6, 64, "ball", 30000, 1, "fp64", "moving"),
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi], mostly odd ones."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.7 else n


def draw(rng):
    family = rng.choice(["laplace", "laplace", "laplace_mixed", "laplace_mixed", "vector", "vector_mixed", "grad",
                         "moving"])
    pts = rng.choice([40, 64, 100, 150])
    points = rng.choice(["uniform", "sphere_clusters", "sphere", "ellipsoids", "shell", "ball"])
    if family == "laplace":
        n = _log(rng, 2000, 300000)
        return _case(None, rng.choice([111, 111, 121]), rng.randint(3, 7), pts, points, n, rng.choice([1, 1, 1, 2, 3]),
                     "fp64", rng.choice(["device", "graph"]), n_trg=rng.choice([0, 0, n // 2 + 1]))
    if family == "laplace_mixed":
        n = _log(rng, 2000, 300000)
        return _case(None, rng.choice([111, 111, 121, 312, 322]), rng.randint(3, 8), pts, points, n,
                     rng.choice([1, 2, 3, 4, 5, 8, 8, 11, 16]), "mixed", rng.choice(["device", "graph"]),
                     n_trg=rng.choice([0, 0, n // 2 + 1]))
    if family == "vector":
        n = _log(rng, 2000, 60000)
        return _case(None, rng.choice([311, 321, 511, 521]), rng.randint(3, 6), pts, points, n, 1, "fp64",
                     rng.choice(["device", "host"]), nu=0.3)
    if family == "vector_mixed":
        n = _log(rng, 2000, 100000)
        return _case(None, rng.choice([311, 321, 511, 521]), rng.randint(4, 8), pts, points, n,
                     rng.choice([1, 2, 4, 5, 8]), "mixed", "device", n_trg=rng.choice([0, 0, n // 3 + 2]), nu=0.3)
    if family == "grad":
        return _case(None, rng.choice([111, 121]), rng.randint(4, 6), pts, points, _log(rng, 4000, 130000),
                     rng.choice([1, 2]), rng.choice(["fp64", "mixed"]), "grad")
    return _case(None, 311, rng.choice([4, 6]), 64, "ball", _log(rng, 3000, 60000), 1, rng.choice(["fp64", "mixed"]),
                 "moving")


def _points(kind, n, rng):
    """(positions, unit normals) in the unit box."""
    if kind == "ellipsoids":
        return workloads.ellipsoids(n, rng)
    if kind == "uniform":
        p = workloads.uniform(n, rng)
    elif kind == "sphere_clusters":
        p = workloads.sphere_clusters(n, rng)
    elif kind == "sphere":
        p = workloads.sphere(n, rng)
        return p, (p - 0.5) / np.linalg.norm(p - 0.5, axis=1)[:, None]
    elif kind == "shell":  # 70 % uniform, 30 % on a thin shell
        m = int(0.7 * n)
        v = workloads.unit_normals(rng, n - m)
        p = np.concatenate([workloads.uniform(m, rng), 0.5 + rng.uniform(0.299, 0.301, size=(n - m, 1)) * v])
    else:  # "ball": the droplets' cloud in the frame of the evaluator's box
        v = workloads.unit_normals(rng, n) * np.cbrt(rng.random((n, 1)))
        p = 0.5 + 0.49 * v
    return p, workloads.unit_normals(rng, n)


def _host_inputs(case, seed):
    """Source positions, normals, targets (None: the sources), densities [k, n, srcDOF], weights [k, n_trg, trgDOF]."""
    rng = np.random.default_rng([workloads.SEED, seed])
    n, k = case["n"], case["k"]
    sd, td = fmmg.KERNELS[case["kernel"]]
    src, nrm = _points(case["points"], n, rng)
    trg = workloads.uniform(case["n_trg"], rng) if case["n_trg"] else None
    den = rng.normal(size=(k, n, sd))
    w = rng.normal(size=(k, n if trg is None else len(trg), td))
    return src, nrm, trg, den, w


_STREAM = []


def _stream():
    """The program's torch stream, which every handle of this process shares."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def prepare(case, seed):
    src, nrm, trg, den, w = _host_inputs(case, seed)
    prec = fmmg.PREC_FP64 if case["precision"] == "fp64" else fmmg.PREC_MIXED
    s = dict(call=case["call"], prec=prec, k=case["k"])
    if case["call"] == "moving":
        s["vel"] = droplets.FmmVelocity(case["np"], case["pts_max"], prec)
        s["x"] = torch.from_numpy(src).cuda()
        s["den"] = torch.from_numpy(den).cuda().view(-1)
        return s
    own = case["call"] in ("device", "graph")
    f = fmmg.FMM3d(case["kernel"], np_=case["np"], pts_max=case["pts_max"], coefs=(1.0, case["nu"]),
                   stream=_stream().cuda_stream if own else None)
    f.setup(src, nrm if case["kernel"] in NORMALS else None, trg)
    s["f"] = f
    if case["call"] == "host":
        f.set_precision(prec)
        s["den"] = den[0]
        return s
    s["den"] = torch.from_numpy(den).cuda()
    if case["call"] == "grad":
        s["den"].requires_grad_(True)
        s["trg"] = torch.from_numpy(src if trg is None else trg).cuda().requires_grad_(True)
        s["w"] = torch.from_numpy(w).cuda()
        return s
    s["out"] = torch.empty(w.shape, dtype=torch.float64, device="cuda")
    f.set_graph(case["call"] == "graph")
    return s


def run(s):
    call = s["call"]
    if call == "moving":
        return s["vel"](s["x"], s["den"])
    f = s["f"]
    if call == "host":
        return f.evaluate(s["den"])
    if call == "grad":
        val = fmmg_torch.fmm_apply(f, s["den"], s["trg"], s["prec"])
        g_den, g_trg = torch.autograd.grad(val, (s["den"], s["trg"]), s["w"])
        return {"val": val.detach(), "grad_den": g_den, "grad_trg": g_trg}
    f.evaluate_device(s["den"], s["out"], s["k"], s["prec"])
    return s["out"]


def work(case):
    """Positions (and normals) and densities read once and values written
    once; the FMM's kernel sums, equivalent-density products and spectral
    translations for a tree whose leaves hold 0.45 pts_max points, 27
    near leaves and 189 V-list boxes a leaf at most (a filled octree; surface
    point sets have fewer)."""
    sd, td = fmmg.KERNELS[case["kernel"]]
    n, k, p = case["n"], case["k"], case["np"]
    nt = case["n_trg"] or n
    esd, etd = {1: (1, 1), 3: (4, 3) if case["kernel"] < 500 else (3, 3)}[td]
    near = 12.0 * case["pts_max"]
    surf, leaves = 6 * (p - 1) ** 2 + 2, n / (0.45 * case["pts_max"])
    chk = 6 * (p + 1) ** 2 + 2
    freq = (2 * p - 1) ** 2 * p
    pairs = nt * near * (11 + 2 * sd * td * k) + n * chk * (11 + 2 * sd * etd * k) + nt * surf * (11 + 2 * esd * td * k)
    gemm = 2.0 * k * leaves * (surf * esd) * ((chk + 2 * surf) * etd + 2 * surf * esd)
    m2l = 8.0 * k * leaves * 90 * freq * esd * etd
    vec = 8.0 * k * (n * sd + nt * td)
    pos = 24.0 * (n + (case["n_trg"] or 0) + (n if case["kernel"] in NORMALS else 0))
    times = 3.0 if case["call"] == "grad" else 1.0
    grad = vec + 24.0 * nt if case["call"] == "grad" else 0.0
    return {"bytes": pos + vec + grad, "flops": times * (pairs + gemm + m2l)}


# About four times the largest difference measured over listed and drawn cases
# between orders of summation (points given in another order; in the mixed
# form also the row GEMMs on CUDA cores in place of the split tensor-core
# products).  It grows with np because the check-to-equivalent
# pseudo-inverse, cut off at 10^-(np+1), amplifies rounding.
_FP64_TOL = {3: 2e-13, 4: 2e-12, 5: 2e-11, 6: 1.4e-10, 7: 5e-10}
_MIXED_TOL = {3: 1.5e-6, 4: 7e-6, 5: 1.4e-5, 6: 1.4e-5, 7: 2e-5, 8: 2e-5}


def tolerance(case):
    if case["precision"] == "fp64":
        return {"rel": _FP64_TOL[case["np"]]}
    if case["kernel"] in NORMALS and case["np"] >= 7:
        # double layers of smooth closed surfaces cancel: 2.5e-5 seen
        return {"rel": 1e-4}
    return {"rel": _MIXED_TOL[case["np"]]}


# ---------------------------------------------------------------- 64-bit sums
def _entries(kt, nu, d, r2, nrm):
    """{(t, s): matrix} of the kernel blocks for offsets d = x - y (three
    [targets, sources] matrices), unit viscosity / shear modulus; a pair with
    r < 1e-8 adds nothing."""
    ir = torch.where(r2 < 1e-16, torch.zeros_like(r2), r2.rsqrt())
    ir2 = ir * ir
    ir3 = ir2 * ir
    pi = math.pi
    rn = None if nrm is None else d[0] * nrm[:, 0] + d[1] * nrm[:, 1] + d[2] * nrm[:, 2]
    if kt == 111:
        return {(0, 0): ir / (4 * pi)}
    if kt == 121:
        return {(0, 0): rn * ir3 / (-4 * pi)}
    if kt == 312:
        return {(0, s): d[s] * ir3 / (4 * pi) for s in range(3)}
    if kt == 322:
        return {(0, s): (nrm[:, s] - 3 * rn * d[s] * ir2) * ir3 / (2 * pi) for s in range(3)}
    out = {}
    for t in range(3):
        for s in range(3):
            if kt == 311:
                m = d[t] * d[s] * ir2 * ir / (8 * pi)
                out[t, s] = m + ir / (8 * pi) if s == t else m
            elif kt == 321:
                out[t, s] = rn * ir3 * ir2 * d[t] * d[s] * (-6 / (8 * pi))
            elif kt == 511:
                c = 1 / (16 * pi * (1 - nu))
                m = d[t] * d[s] * ir3 * c
                out[t, s] = m + (3 - 4 * nu) * c * ir if s == t else m
            else:  # 521
                a = (1 - 2 * nu) / (8 * pi * (1 - nu))
                m = (d[t] * nrm[:, s] - nrm[:, t] * d[s]) * a * ir3 - 3 / (8 * pi * (1 - nu)) * rn * ir3 * ir2 * d[t] * d[s]
                out[t, s] = m - a * rn * ir3 if s == t else m
    return out


def exact(case, seed):
    """The dense sums in 64 bits (and, for gradients, their transposes and
    derivatives).  None where they would take over 20 seconds."""
    n, nt, k = case["n"], case["n_trg"] or case["n"], case["k"]
    if n * nt > 1.5e11:
        return None
    src, nrm, trg, den, w = _host_inputs(case, seed)
    kt = case["kernel"]
    sd, td = fmmg.KERNELS[kt]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    y = torch.from_numpy(src).to(dev)
    x = y if trg is None else torch.from_numpy(trg).to(dev)
    q = torch.from_numpy(nrm).to(dev) if kt in NORMALS else None
    dt = torch.from_numpy(den).to(dev)
    wt = torch.from_numpy(w).to(dev)
    col = [dt[:, :, s].t().contiguous() for s in range(sd)]  # [n, k]
    val = torch.zeros(nt, td, k, dtype=torch.float64, device=dev)
    grad = case["call"] == "grad"
    g_den = torch.zeros(k, n, dtype=torch.float64, device=dev)
    g_trg = torch.zeros(nt, 3, dtype=torch.float64, device=dev)
    rows = max(1, int(3e7 // n))
    for i in range(0, nt, rows):
        xi = x[i:i + rows]
        d = [xi[:, c:c + 1] - y[:, c] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        for (t, s), m in _entries(kt, case["nu"], d, r2, q).items():
            val[i:i + rows, t] += m @ col[s]
            if grad:
                g_den += wt[:, i:i + rows, 0] @ m
        if grad:  # d/dx of sum_k w_k(x) sum_y K(x - y) den_k(y), kernels 111 and 121
            c = wt[:, i:i + rows, 0].t() @ dt[:, :, 0]
            ir = torch.where(r2 < 1e-16, torch.zeros_like(r2), r2.rsqrt())
            ir3 = ir * ir * ir
            if kt == 111:
                c *= ir3 / (-4 * math.pi)
                for a in range(3):
                    g_trg[i:i + rows, a] = (c * d[a]).sum(1)
            else:
                c *= ir3 / (-4 * math.pi)
                e = c * (d[0] * q[:, 0] + d[1] * q[:, 1] + d[2] * q[:, 2]) * ir * ir * -3
                for a in range(3):
                    g_trg[i:i + rows, a] = c @ q[:, a] + (e * d[a]).sum(1)
    val = val.permute(2, 0, 1).contiguous()
    if grad:
        return {"val": val, "grad_den": g_den.view(k, n, 1), "grad_trg": g_trg}
    if case["call"] in ("host", "moving"):
        return val[0]
    return val
