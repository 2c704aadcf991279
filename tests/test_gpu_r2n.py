"""FP32 + refinement at lengths other than 512 (paired chunks, windows above
512 rows): every place of the last row in its chunk, chunk and window counts,
both layouts, aligned (TMA) and not, in place and out of place, partial groups
of systems, planes.  Tolerance: the refinement tolerance of the other tests,
1e-12 relative (a sweep leaves ~1e-14; the double-word keeps 47 bits)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COMPACT = (1., 2., .25, 1., .25, 2., 1.)
HEAT = (1., 0., -.5, 2., -.5, 0., 1.)
GENERAL = (1.3, .2, -.17, 1.1, .23, .3, .9)
TOL = 1e-12
MANY = 2437  # enough 16-system groups for every SM, the last one partial


def _check(oracle, got, d, n, co):
    pick = np.r_[0:20, len(d) // 2:len(d) // 2 + 5, len(d) - 20:len(d)]
    assert oracle.rel_err(got[pick], oracle.exact_solve(np.ascontiguousarray(d[pick]), n, co)) < TOL
    assert np.isfinite(got).all()


@pytest.mark.parametrize("co", [HEAT, COMPACT, GENERAL], ids=["heat", "compact", "general"])
@pytest.mark.parametrize("n", [64, 65, 66, 79, 80, 81, 100, 240, 241, 385, 496, 500, 511, 513, 576, 700, 1000, 1024,
                               1025, 2048, 2501])
def test_contiguous(cuda, oracle, co, n):
    import ntk

    d = np.random.default_rng(n).normal(size=(MANY, n))
    t = torch.from_numpy(d).to(cuda)
    out = torch.empty_like(t)
    with ntk.Plan(n, MANY, co, precision="fp32_refine") as p:
        p.solve_strided(t, out, MANY, MANY, n, 0, 1)
        p.solve(t)
        assert p.status() == 0
    _check(oracle, out.cpu().numpy(), d, n, co)
    _check(oracle, t.cpu().numpy(), d, n, co)


@pytest.mark.parametrize("co", [HEAT, GENERAL], ids=["heat", "general"])
@pytest.mark.parametrize("n", [64, 95, 97, 385, 512, 700, 1500])
@pytest.mark.parametrize("planes,ni,es", [(1, MANY, 2440), (1, MANY, 2441), (5, 500, 500), (7, 333, 333)])
def test_strided(cuda, oracle, co, n, planes, ni, es):
    """In and out of place; elements beyond a plane's systems are not touched."""
    import ntk

    d = np.random.default_rng(n).normal(size=(planes, n, es))
    t = torch.from_numpy(d).to(cuda)
    out = torch.full_like(t, 3.0)
    with ntk.Plan(n, 0, co, precision="fp32_refine") as p:
        p.solve_strided(t, out, planes * ni, ni, 1, n * es, es)
        p.solve_strided(t, t, planes * ni, ni, 1, n * es, es)
        assert p.status() == 0
    lines = np.moveaxis(d[:, :, :ni], 1, 2).reshape(-1, n)
    for o, rest in ((out.cpu().numpy(), 3.0), (t.cpu().numpy(), d[:, :, ni:])):
        assert (o[:, :, ni:] == rest).all()
        _check(oracle, np.moveaxis(o[:, :, :ni], 1, 2).reshape(-1, n), lines, n, co)


@pytest.mark.parametrize("n", [64, 81, 240, 385, 497, 600, 1025, 2047])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("width", [52, 53])
def test_compact_derivative(cuda, oracle, n, axis, width):
    import ntk

    shape = [width, width, width]
    shape[axis] = n
    f = np.random.default_rng(n).normal(size=shape)
    ft = torch.from_numpy(f).to(cuda)
    out = torch.empty_like(ft)
    h = 1. / (n - 1)
    with ntk.Plan(n, 0, COMPACT, precision="fp32_refine") as p:
        p.compact_deriv(ft, out, axis, h)
        p.compact_deriv(ft, ft, axis, h)
        assert p.status() == 0
    lines = np.ascontiguousarray(np.moveaxis(f, axis, 2)).reshape(-1, n)
    rhs = np.empty_like(lines)
    rhs[:, 1:-1] = 3 / (4 * h) * (lines[:, 2:] - lines[:, :-2])
    rhs[:, 0] = (-5 * lines[:, 0] + 4 * lines[:, 1] + lines[:, 2]) / (2 * h)
    rhs[:, -1] = (5 * lines[:, -1] - 4 * lines[:, -2] - lines[:, -3]) / (2 * h)
    for o in (out, ft):
        _check(oracle, np.moveaxis(o.cpu().numpy(), axis, 2).reshape(-1, n), rhs, n, COMPACT)


def test_out_of_range_input_is_reported(cuda):
    import ntk

    n = 300
    t = torch.ones((MANY, n), dtype=torch.float64, device=cuda)
    t[MANY - 1, 17] = 2.0 ** 130
    with ntk.Plan(n, MANY, HEAT, precision="fp32_refine") as p:
        p.solve(t)
        assert p.status(raise_on_error=False) & 1
        assert p.status() == 0
