"""The work that users of this framework have it do, as cases to be timed.

Every case goes through the public entry points of the ntk package (the
compact derivatives of experiments/run-compact.py, NearToeplitzSolver.solve
of neato.py, the ADI stepper of experiments/run-adi.py, uneven batches), over
sizes from a single small 2D field to a 512^3 field and in all three
precisions.  Systems that are solved in place again and again are implicit
diffusion steps (rows that sum to one), whose values stay in range however
often a pass is repeated.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "near-toeplitz-applications_gb300"))

COMPACT = (1., 2., 1. / 4, 1., 1. / 4, 2., 1.)  # experiments/run-compact.py:48


def listed():
    return [
        # the reference's 2D example field: 256 x 256, one derivative; latency counts
        {"name": "deriv2d_256_f64", "kind": "deriv", "nz": 1, "ny": 256, "nx": 256, "axis": 2, "precision": "fp64"},
        # the headline: all three derivatives of a 512^3 field, in both precisions that reach 1e-12
        {"name": "grad_512_f64", "kind": "grad", "nz": 512, "ny": 512, "nx": 512, "precision": "fp64"},
        {"name": "grad_512_refine", "kind": "grad", "nz": 512, "ny": 512, "nx": 512, "precision": "fp32_refine"},
        # fields as simulations have them, no extent a power of two
        {"name": "grad_ragged_f64", "kind": "grad", "nz": 190, "ny": 333, "nx": 421, "precision": "fp64"},
        {"name": "grad_ragged_refine", "kind": "grad", "nz": 240, "ny": 385, "nx": 700, "precision": "fp32_refine"},
        # a wide slab along one axis in FP32 only, for previews and preconditioners
        {"name": "deriv_y_512_fp32", "kind": "deriv", "nz": 96, "ny": 512, "nx": 640, "axis": 1, "precision": "fp32"},
        # the drop-in solver on the reference's largest system: few systems (one ADI sweep's worth) and many
        {"name": "solve_2048_f64", "kind": "solve", "n": 2048, "nrhs": 2046, "r": 0.5, "precision": "fp64"},
        {"name": "solve_2048_refine", "kind": "solve", "n": 2048, "nrhs": 16384, "r": 0.5,
         "precision": "fp32_refine"},
        # heat equation: a long run on the large grid, and single-digit steps on a grid of odd size
        {"name": "adi_2048_refine", "kind": "adi", "N": 2048, "ratio": 1.0, "steps": 20, "graph": True,
         "precision": "fp32_refine"},
        {"name": "adi_999_f64", "kind": "adi", "N": 999, "ratio": 1.0, "steps": 4, "graph": False,
         "precision": "fp64"},
        # many systems of their own lengths and coefficients in one buffer
        {"name": "batch_4096_refine", "kind": "batch", "count": 4096, "nmin": 32, "nmax": 8192,
         "precision": "fp32_refine"},
        {"name": "batch_1000_f64", "kind": "batch", "count": 1000, "nmin": 17, "nmax": 5000, "precision": "fp64"},
    ]


def _log(rng, lo, hi):
    """A whole number in lo .. hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """As _log, but a power of two one time in three."""
    n = _log(rng, lo, hi)
    if rng.random() < 1 / 3:
        n = max(lo, min(hi, 1 << int(round(math.log2(n)))))
    return n


def draw(rng):
    kind = rng.choice(["deriv", "grad", "grad", "solve", "solve", "adi", "batch"])
    wide = rng.choice(["fp64", "fp32_refine"])
    if kind == "deriv":  # 2D fields and slabs
        nz, ny, nx = rng.choice([1, 1, _log(rng, 2, 100)]), _size(rng, 64, 1024), _size(rng, 64, 1024)
        return {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "axis": rng.choice([1, 2]),
                "precision": rng.choice(["fp64", "fp32_refine", "fp32"])}
    if kind == "grad":
        return {"kind": kind, "nz": _size(rng, 32, 512), "ny": _size(rng, 32, 512), "nx": _size(rng, 32, 512),
                "precision": wide}
    if kind == "solve":
        n = _size(rng, 32, 4096)
        return {"kind": kind, "n": n, "nrhs": _log(rng, 64, min(65536, (1 << 26) // n)),
                "r": rng.choice([0.5, 0.5, 1.0, 0.3]), "precision": wide}
    if kind == "adi":
        return {"kind": kind, "N": _size(rng, 128, 2048), "ratio": rng.choice([1.0, 1.0, 0.5, 2.0]),
                "steps": rng.randint(1, 20), "graph": rng.random() < 0.5, "precision": wide}
    return {"kind": kind, "count": _log(rng, 64, 4096), "nmin": rng.randint(16, 64), "nmax": _log(rng, 512, 8192),
            "precision": wide}


# ---- inputs, from the case and the seed alone ------------------------------


def _field(shape, seed):
    """Eight random Fourier modes on the unit cube, as the reference's analytic test fields."""
    rng = np.random.default_rng(seed)
    f = torch.zeros(shape, dtype=torch.float64, device="cuda")
    axes = [torch.linspace(0, 1, s, dtype=torch.float64, device="cuda") for s in shape]
    for _ in range(8):
        k, phase, amp = rng.integers(1, 17, size=len(shape)), rng.random(), rng.normal()
        arg = 2 * math.pi * phase
        for d, ax in enumerate(axes):
            arg = arg + (2 * math.pi * float(k[d])) * ax.view([-1 if e == d else 1 for e in range(len(shape))])
        f += amp * torch.sin(arg)
    return f


def _noise(shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _axes(case):
    """(axis, extent, grid spacing) of each derivative that the case takes, x first."""
    ext = (case["nz"], case["ny"], case["nx"])
    return [(a, ext[a], 1. / (ext[a] - 1)) for a in ((2, 1, 0) if case["kind"] == "grad" else (case["axis"],))]


def _heat(case):
    """Backward Euler for the heat equation on a line, fixed ends."""
    r = case["r"]
    return (1., 0., -r, 1. + 2. * r, -r, 0., 1.)


def _plate(case, seed):
    """Sixteen warm spots on a plate whose edges are held at one."""
    N = case["N"]
    rng = np.random.default_rng(seed)
    g = torch.linspace(0, 1, N, dtype=torch.float64, device="cuda")
    u = torch.zeros((N, N), dtype=torch.float64, device="cuda")
    for _ in range(16):
        (cx, cy), w = rng.random(2), rng.uniform(0.02, 0.1)
        u += torch.exp(-(g[:, None] - cy) ** 2 / (2 * w * w)) * torch.exp(-(g[None, :] - cx) ** 2 / (2 * w * w))
    u[0, :] = u[-1, :] = 0
    u[:, 0] = u[:, -1] = 0
    return u + 1.


def _lines(case, seed):
    """Lengths and rows (a, b, c) of implicit diffusion on lines of their own length and diffusivity.  The
    lengths, and with them the buffer's size, are the case's; the rows are the seed's."""
    count = case["count"]
    n = np.exp(np.random.default_rng(count).uniform(math.log(case["nmin"]), math.log(case["nmax"]), size=count))
    n = np.clip(n.astype(np.int32), case["nmin"], case["nmax"])
    rng = np.random.default_rng(seed)

    def rows(shape, lo, hi):
        a, c = -rng.uniform(lo, hi, size=shape), -rng.uniform(lo, hi, size=shape)
        return np.stack([a, 1. - a - c, c], axis=-1)

    interior, head, tail = rows(count, 0.2, 0.75), rows((count, 2), 0., 0.4), rows((count, 2), 0., 0.4)
    head[:, 0, 1] += head[:, 0, 0]
    head[:, 0, 0] = 0
    tail[:, 1, 1] += tail[:, 1, 2]
    tail[:, 1, 2] = 0
    return n, interior, head, tail


# ---- one pass ---------------------------------------------------------------


def prepare(case, seed):
    import ntk
    from neato import NearToeplitzSolver

    kind, prec = case["kind"], case["precision"]
    if kind in ("deriv", "grad"):
        f = _field((case["nz"], case["ny"], case["nx"]), seed)
        plans = {}
        for _, n, _ in _axes(case):
            if n not in plans:
                plans[n] = ntk.Plan(n, 0, COMPACT, precision=prec)
        work = [(plans[n], axis, h, torch.empty_like(f)) for axis, n, h in _axes(case)]
        return {"kind": kind, "f": f, "work": work}
    if kind == "solve":
        solver = NearToeplitzSolver(case["n"], case["nrhs"], _heat(case), precision=prec, strict=False)
        return {"kind": kind, "solver": solver, "d": _noise((case["nrhs"], case["n"]), seed)}
    if kind == "adi":
        N = case["N"]
        dx = 1. / (N - 1)
        u = _plate(case, seed)
        return {"kind": kind, "adi": ntk.Adi(N, dx, case["ratio"] * dx * dx, precision=prec), "u": u,
                "d_x": u.clone(), "d_y": u.t().contiguous(), "steps": case["steps"], "graph": case["graph"]}
    n, interior, head, tail = _lines(case, seed)
    return {"kind": kind, "batch": ntk.UnevenBatch(n, interior, head, tail, precision=prec),
            "d": _noise(int(n.sum()), seed)}


def run(state):
    kind = state["kind"]
    if kind in ("deriv", "grad"):
        for plan, axis, h, out in state["work"]:
            plan.compact_deriv(state["f"], out, axis, h)
        return [w[3] for w in state["work"]]
    if kind == "solve":
        state["solver"].solve(state["d"])
        return state["d"]
    if kind == "adi":
        state["adi"].run(state["u"], state["d_x"], state["d_y"], state["steps"], graph=state["graph"])
        return {"u": state["u"], "d_x": state["d_x"]}
    state["batch"].solve(state["d"])
    return state["d"]


# ---- what a pass cannot do without ------------------------------------------


def work(case):
    """Each input read once and each output written once; two multiply-adds and a multiply per unknown for the
    sweeps, and the right-hand side's own operations."""
    kind = case["kind"]
    if kind in ("deriv", "grad"):
        points, outs = case["nz"] * case["ny"] * case["nx"], len(_axes(case))
        return {"bytes": 8. * points * (1 + outs), "flops": 6. * points * outs}
    if kind == "solve":
        rows = case["n"] * case["nrhs"]
        return {"bytes": 16. * rows, "flops": 5. * rows}
    if kind == "adi":
        rows = case["N"] ** 2
        return {"bytes": 24. * rows, "flops": 2 * 10. * rows * case["steps"]}
    mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    return {"bytes": 16. * case["count"] * mean, "flops": 5. * case["count"] * mean}


# ---- the same in plain 64-bit arithmetic ---------------------------------------


def _thomas(a, b, c, d):
    """Tridiagonal systems down the first axis of d; a, b, c per row (numbers, or tensors over the systems)."""
    n = d.shape[0]
    d = d.clone()
    u = [b[0]]
    for i in range(1, n):
        m = a[i] / u[i - 1]
        u.append(b[i] - m * c[i - 1])
        d[i] -= m * d[i - 1]
    d[n - 1] /= u[n - 1]
    for i in range(n - 2, -1, -1):
        d[i] = (d[i] - c[i] * d[i + 1]) / u[i]
    return d


def _rows(coeffs, n):
    b1, c1, ai, bi, ci, an, bn = coeffs
    return [0.] + [ai] * (n - 2) + [an], [b1] + [bi] * (n - 2) + [bn], [c1] + [ci] * (n - 2) + [0.]


def _exact_deriv(f, axis, h):
    g = f.movedim(axis, 0).contiguous()
    d = torch.empty_like(g)
    d[1:-1] = (3. / (4 * h)) * (g[2:] - g[:-2])
    d[0] = (-5 * g[0] + 4 * g[1] + g[2]) / (2 * h)
    d[-1] = (5 * g[-1] - 4 * g[-2] - g[-3]) / (2 * h)
    return _thomas(*_rows(COMPACT, g.shape[0]), d).movedim(0, axis).contiguous()


def _exact_adi(case, seed):
    """experiments/run-adi.py:59-71 with whole-array stencils; its rows are lines down the first axis here."""
    N = case["N"]
    dx = 1. / (N - 1)
    dt = case["ratio"] * dx * dx
    rows = _rows((1., 0., 1 / dx ** 2, -2 * (1 / dt + 1 / dx ** 2), 1 / dx ** 2, 0., 1.), N)
    u = _plate(case, seed)
    d_x, d_y = u.clone(), u.t().contiguous()
    for _ in range(case["steps"]):
        for d in (d_x, d_y):
            d[1:-1, 1:-1] = (2 * (1 / dx ** 2 - 1 / dt) * u[1:-1] - (u[:-2] + u[2:]) / dx ** 2)[:, 1:-1]
            d[1:-1] = _thomas(*rows, d[1:-1].t().contiguous()).t()
            u = d.t().contiguous()
    return {"u": u, "d_x": d_x}


def _exact_batch(case, seed):
    n, interior, head, tail = _lines(case, seed)
    count, most = len(n), int(n.max())
    offset = np.concatenate([[0], np.cumsum(n.astype(np.int64))])
    row, last = np.arange(most)[:, None], n[None, :].astype(np.int64)
    m = [np.where(row < last, interior[None, :, k], 1. if k == 1 else 0.) for k in range(3)]
    every = np.arange(count)
    for k in range(3):
        for j in range(2):
            m[k][j, :] = head[:, j, k]
            m[k][n - 2 + j, every] = tail[:, j, k]
    a, b, c = (torch.from_numpy(x).cuda() for x in m)
    inside = torch.from_numpy(row < last).cuda()
    at = torch.from_numpy(np.where(row < last, offset[:-1][None, :] + row, 0)).cuda()
    d = _noise(int(n.sum()), seed)
    x = _thomas(a, b, c, torch.where(inside, d[at], torch.zeros((), dtype=torch.float64, device="cuda")))
    out = torch.empty_like(d)
    out[at[inside]] = x[inside]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("deriv", "grad"):
        f = _field((case["nz"], case["ny"], case["nx"]), seed)
        return [_exact_deriv(f, axis, h) for axis, _, h in _axes(case)]
    if kind == "solve":
        d = _noise((case["nrhs"], case["n"]), seed)
        return _thomas(*_rows(_heat(case), case["n"]), d.t().contiguous()).t().contiguous()
    if kind == "adi":
        return _exact_adi(case, seed)
    return _exact_batch(case, seed)
