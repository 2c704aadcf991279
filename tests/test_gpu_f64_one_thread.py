"""FP64 with one thread per system, forced: every launch variant of the
contiguous sweeps and the strided one, at lengths that leave remainders in the
row blocks (8) and tiles (16) and system counts that leave partial warps.
Tolerance: FP64 throughout, matrices with |A^-1| |A| <= 50 and up to 16
roundings a row: 50 * 16 * 2^-53 ~ 1e-13 of the long-double solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COMPACT = (1., 2., .25, 1., .25, 2., 1.)
HEAT = (1., 0., -.5, 2., -.5, 0., 1.)
TOL = 1e-13
SIZES = [4, 8, 9, 15, 16, 17, 18, 23, 24, 25, 33, 41, 48, 49, 65, 100, 129, 161, 257, 333, 513, 700]


def _rhs(lines, h):
    rhs = np.empty_like(lines)
    rhs[:, 1:-1] = 3 / (4 * h) * (lines[:, 2:] - lines[:, :-2])
    rhs[:, 0] = (-5 * lines[:, 0] + 4 * lines[:, 1] + lines[:, 2]) / (2 * h)
    rhs[:, -1] = (5 * lines[:, -1] - 4 * lines[:, -2] - lines[:, -3]) / (2 * h)
    return rhs


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("nsys", [1, 45, 129])
def test_contiguous(cuda, oracle, variant, n, nsys):
    import ntk

    d = np.random.default_rng(n + nsys).normal(size=(nsys, n))
    h = 1. / (n - 1)
    t = torch.from_numpy(d).to(cuda)
    out, f, g = torch.empty_like(t), t.view(1, nsys, n).clone(), torch.empty_like(t).view(1, nsys, n)
    with ntk.Plan(n, nsys, HEAT) as p, ntk.Plan(n, 0, COMPACT) as q:
        for plan in (p, q):
            plan.set_tuning(f64_x_variant=variant)
            assert plan.get_tuning()["f64_chunks"] == 1
        p.solve_strided(t, out, nsys, nsys, n, 0, 1)
        p.solve(t)
        q.compact_deriv(f, g, 2, h)
        q.compact_deriv(f, f, 2, h)
    want = oracle.exact_solve(d, n, HEAT)
    assert oracle.rel_err(out.cpu().numpy(), want) < TOL
    assert oracle.rel_err(t.cpu().numpy(), want) < TOL
    want = oracle.exact_solve(_rhs(d, h), n, COMPACT)
    assert oracle.rel_err(g[0].cpu().numpy(), want) < TOL
    assert oracle.rel_err(f[0].cpu().numpy(), want) < TOL


@pytest.mark.parametrize("threads", [32, 64, 128])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("planes,ni", [(1, 77), (3, 35)])
def test_strided(cuda, oracle, threads, n, planes, ni):
    import ntk

    d = np.random.default_rng(n + ni).normal(size=(planes, n, ni))
    h = 1. / (n - 1)
    t = torch.from_numpy(d).to(cuda)
    out, f, g = torch.empty_like(t), t.clone(), torch.empty_like(t)
    with ntk.Plan(n, 0, HEAT) as p, ntk.Plan(n, 0, COMPACT) as q:
        for plan in (p, q):
            plan.set_tuning(f64_threads=threads)
        p.solve_strided(t, out, planes * ni, ni, 1, n * ni, ni)
        p.solve_strided(t, t, planes * ni, ni, 1, n * ni, ni)
        q.compact_deriv(f, g, 1, h)
        q.compact_deriv(f, f, 1, h)
    lines = np.ascontiguousarray(np.moveaxis(d, 1, 2)).reshape(-1, n)
    for got, want in ((out, oracle.exact_solve(lines, n, HEAT)), (t, oracle.exact_solve(lines, n, HEAT)),
                      (g, oracle.exact_solve(_rhs(lines, h), n, COMPACT)),
                      (f, oracle.exact_solve(_rhs(lines, h), n, COMPACT))):
        assert oracle.rel_err(np.moveaxis(got.cpu().numpy(), 1, 2).reshape(-1, n), want) < TOL


def test_the_keys_choose_the_kernel(cuda):
    """70 systems of 700 rows: by the rule several threads each, whose carries
    round differently somewhere; a one-thread key takes the one-thread kernel,
    and f64_chunks either, whatever was set before."""
    import ntk

    d = torch.from_numpy(np.random.default_rng(3).normal(size=(70, 700))).to(cuda)

    def solved(**tuning):
        t = d.clone()
        with ntk.Plan(700, 70, HEAT) as p:
            p.set_tuning(**tuning)
            p.solve(t)
        return t

    one, many = solved(f64_chunks=1), solved(f64_chunks=2)
    assert not torch.equal(one, many)
    assert torch.equal(solved(), many)
    for key in ({"f64_x_variant": 0}, {"f64_x_variant": 1}, {"f64_x_variant": 2}, {"f64_threads": 128}):
        assert torch.equal(solved(**key), one), key
        assert torch.equal(solved(f64_chunks=2, **key), many), key
    with ntk.Plan(700, 70, HEAT) as p:
        with pytest.raises(ValueError):
            p.set_tuning(f64_chunks=3)
