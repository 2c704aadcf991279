"""FP64 solves of few systems (several threads per system): sizes around the
chunk boundaries, both layouts, slowly decaying factors, and systems with
values that are not finite.

Tolerance: the solves are FP64 throughout with three roundings a row more
than a sequential Thomas solve at most; every matrix here has
|A^-1| |A| <= 50, so the result stays within 50 * 16 * 2^-53 ~ 1e-13 of the
long-double solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COMPACT = (1., 2., .25, 1., .25, 2., 1.)
HEAT = (1., 0., -.5, 2., -.5, 0., 1.)
SLOW = (3., 1., -4., 9., -4., .5, 2.)  # multipliers 0.61: carries reach far
TOL = 1e-13


@pytest.mark.parametrize("coeffs", [COMPACT, HEAT, SLOW], ids=["compact", "heat", "slow"])
@pytest.mark.parametrize("n", [17, 20, 21, 36, 63, 64, 65, 129, 257, 999, 2048, 4097, 9001, 20001])
@pytest.mark.parametrize("nsys", [1, 3, 37])
def test_contiguous(cuda, oracle, coeffs, n, nsys):
    import ntk

    d = np.random.default_rng(n + nsys).normal(size=(nsys, n))
    t = torch.from_numpy(d).to(cuda)
    with ntk.Plan(n, nsys, coeffs) as p:
        p.solve(t)
    assert oracle.rel_err(t.cpu().numpy(), oracle.exact_solve(d, n, coeffs)) < TOL


@pytest.mark.parametrize("n", [17, 31, 64, 100, 333, 1030])
@pytest.mark.parametrize("planes,ni", [(1, 1), (1, 5), (3, 7), (2, 18)])
def test_strided(cuda, oracle, n, planes, ni):
    """Out of place, planes of ni adjacent systems; rows beyond the systems
    stay as they are."""
    import ntk

    rng = np.random.default_rng(n + ni)
    d = rng.normal(size=(planes, n, ni + 1))
    t = torch.from_numpy(d).to(cuda)
    out = torch.full_like(t, 7.0)
    with ntk.Plan(n, 0, HEAT) as p:
        p.solve_strided(t, out, planes * ni, ni, 1, n * (ni + 1), ni + 1)
    o = out.cpu().numpy()
    assert (o[:, :, ni] == 7.0).all()
    rows = np.ascontiguousarray(np.moveaxis(d[:, :, :ni], 1, 2)).reshape(-1, n)
    got = np.moveaxis(o[:, :, :ni], 1, 2).reshape(-1, n)
    assert oracle.rel_err(got, oracle.exact_solve(rows, n, HEAT)) < TOL


@pytest.mark.parametrize("n", [20, 33, 64, 321, 700])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_compact_derivative(cuda, oracle, n, axis):
    """In place and out of place, against the long-double solve."""
    import ntk

    shape = [3, 5, 4]
    shape[axis] = n
    f = torch.from_numpy(np.random.default_rng(n).normal(size=shape)).to(cuda)
    h = 1. / (n - 1)
    out = torch.empty_like(f)
    with ntk.Plan(n, 0, COMPACT) as p:
        p.compact_deriv(f, out, axis, h)
        g = f.clone()
        p.compact_deriv(g, g, axis, h)
    assert torch.equal(out, g)
    lines = np.ascontiguousarray(np.moveaxis(f.cpu().numpy(), axis, 2)).reshape(-1, n)
    rhs = np.empty_like(lines)
    rhs[:, 1:-1] = 3 / (4 * h) * (lines[:, 2:] - lines[:, :-2])
    rhs[:, 0] = (-5 * lines[:, 0] + 4 * lines[:, 1] + lines[:, 2]) / (2 * h)
    rhs[:, -1] = (5 * lines[:, -1] - 4 * lines[:, -2] - lines[:, -3]) / (2 * h)
    got = np.moveaxis(out.cpu().numpy(), axis, 2).reshape(-1, n)
    assert oracle.rel_err(got, oracle.exact_solve(rhs, n, COMPACT)) < TOL


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan"), 1.5e308])
@pytest.mark.parametrize("strided", [False, True])
def test_not_finite_values_spread_as_in_a_sequential_solve(cuda, bad, strided):
    """One system meets a value that is not finite (or overflows on the way);
    the others are untouched by it."""
    import ntk

    n, ns, at, row = 200, 9, 4, 117
    co = (1., 2., 1., 2.5, -1., 2., 1.)
    d = np.random.default_rng(1).normal(size=(ns, n))
    d[at, row] = bad
    if bad == 1.5e308:
        d[at, row - 1] = -bad
    want = d.copy()
    with np.errstate(all="ignore"):
        l, u = np.zeros(n), np.zeros(n)
        a = np.array([0.] + [co[2]] * (n - 2) + [co[5]])
        b = np.array([co[0]] + [co[3]] * (n - 2) + [co[6]])
        c = np.array([co[1]] + [co[4]] * (n - 2) + [0.])
        u[0] = b[0]
        for i in range(1, n):
            l[i] = a[i] / u[i - 1]
            u[i] = b[i] - l[i] * c[i - 1]
        for i in range(1, n):
            want[:, i] = want[:, i] - l[i] * want[:, i - 1]
        want[:, n - 1] = want[:, n - 1] / u[n - 1]
        for i in range(n - 2, -1, -1):
            want[:, i] = want[:, i] / u[i] - (c[i] / u[i]) * want[:, i + 1]
    t = torch.from_numpy(d.T.copy() if strided else d).to(cuda)
    with ntk.Plan(n, ns, co) as p:
        if strided:
            p.solve_strided(t, t, ns, ns, 1, 0, ns)
        else:
            p.solve(t)
    got = t.cpu().numpy().T if strided else t.cpu().numpy()
    assert not np.isfinite(want[at]).all()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    ok = np.isfinite(want)
    assert np.allclose(got[ok], want[ok], rtol=1e-12, atol=1e-13)
