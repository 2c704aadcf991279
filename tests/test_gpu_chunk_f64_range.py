"""FP64 solves of few systems at the upper end of the range: systems whose
values overflow only once the carry of the rows behind is added, wherever the
overflow lies in its thread's rows, spread inf as a sequential solve does.

x_i = d_i + x_{i+1} / 2 (a = 0, b = 1, c = -1/2): every value below is exact or
far from a rounding that could change which rows are finite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CO = (1., -.5, 0., 1., -.5, 0., 1.)


def _systems(n):
    """System s holds 1.2e308 in row s and 1.7e308 in row s + 1: each is
    finite, 1.2e308 + 1.7e308 / 2 is not."""
    d = np.full((n - 1, n), .125)
    s = np.arange(n - 1)
    d[s, s] = 1.2e308
    d[s, s + 1] = 1.7e308
    return d


def _sequential(d):
    x = d.copy()
    with np.errstate(over="ignore"):
        for i in range(d.shape[1] - 2, -1, -1):
            x[:, i] = d[:, i] + .5 * x[:, i + 1]
    return x


@pytest.mark.parametrize("n", [40, 129, 200])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("in_place", [False, True])
def test_overflow_with_the_carry_spreads(cuda, n, strided, in_place):
    import ntk

    d = _systems(n)
    want = _sequential(d)
    k = n - 1
    assert (np.isinf(want).sum(axis=1) == np.arange(1, n)).all()
    t = torch.from_numpy(d.T.copy() if strided else d).to(cuda)
    out = t if in_place else torch.empty_like(t)
    with ntk.Plan(n, k, CO) as p:
        if strided:
            p.solve_strided(t, out, k, k, 1, 0, k)
        else:
            p.solve_strided(t, out, k, k, n, 0, 1)
    got = out.cpu().numpy().T if strided else out.cpu().numpy()
    assert np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.array_equal(got[~ok], want[~ok])
    assert np.allclose(got[ok], want[ok], rtol=1e-14, atol=0)


@pytest.mark.parametrize("n", [20, 27, 100])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_bad_row_of_a_derivative(cuda, n, bad):
    """A nan or inf anywhere in a line of a compact derivative, in and out of
    place, as in the sequential sweeps of the matrix."""
    import ntk

    co = (1., 2., 1. / 4, 1., 1. / 4, 2., 1.)
    f = np.random.default_rng(n).normal(size=(1, n, n))
    f[0, np.arange(n), np.arange(n)] = bad  # line i is bad in row i
    h = .5
    with np.errstate(all="ignore"):
        g = f[0]
        rhs = np.empty_like(g)
        rhs[:, 1:-1] = g[:, 2:] - g[:, :-2]
        rhs[:, 0] = (-5 * g[:, 0] + 4 * g[:, 1] + g[:, 2]) * (1. / 3 * 2)
        rhs[:, -1] = -(-5 * g[:, -1] + 4 * g[:, -2] + g[:, -3]) * (1. / 3 * 2)
        a = np.array([0.] + [.25] * (n - 2) + [2.])
        c = np.array([2.] + [.25] * (n - 2) + [0.])
        u, l = np.ones(n), np.zeros(n)
        for i in range(1, n):
            l[i] = a[i] / u[i - 1]
            u[i] = 1. - l[i] * c[i - 1]
        for i in range(1, n):
            rhs[:, i] -= l[i] * rhs[:, i - 1]
        x = np.empty_like(rhs)
        x[:, -1] = rhs[:, -1] * (1.5 / u[-1])
        for i in range(n - 2, -1, -1):
            x[:, i] = rhs[:, i] * (1.5 / u[i]) - (c[i] / u[i]) * x[:, i + 1]
    t = torch.from_numpy(f).to(cuda)
    out = torch.empty_like(t)
    with ntk.Plan(n, 0, co) as p:
        p.compact_deriv(t, out, 2, h)
        p.compact_deriv(t, t, 2, h)
    for got in (out.cpu().numpy()[0], t.cpu().numpy()[0]):
        assert np.array_equal(np.isnan(got), np.isnan(x))
        assert np.array_equal(got[np.isinf(x)], x[np.isinf(x)])
