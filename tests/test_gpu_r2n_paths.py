"""FP32 + refinement on paired chunks of any number, forced (refine_kernel =
2): every place of the last row in its chunk with one window and with several,
both layouts, with and without tensor maps and bulk copies, in place and out of
place, many planes; that the forced kernel is the one that runs; and the rule
that leaves small batches with the chunked kernels.  Tolerance: the refinement
tolerance of the other tests, 1e-12 relative."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COMPACT = (1., 2., .25, 1., .25, 2., 1.)
HEAT = (1., 0., -.5, 2., -.5, 0., 1.)
GENERAL = (1.3, .2, -.17, 1.1, .23, .3, .9)
LIMIT = (1., 0., -.7, 2.4, -.7, 0., 1.)  # multipliers 0.322: the slowest decay that is served
TOL = 1e-12
PLACES = list(range(96, 113)) + list(range(513, 530)) + [1025, 1500, 2047]


def _solved(t, out, n, co, layout, kernel):
    import ntk

    with ntk.Plan(n, 0, co, precision="fp32_refine") as p:
        p.set_tuning(refine_kernel=kernel)
        p.solve_strided(t, out, *layout)
        assert p.status() == 0
    return out


@pytest.mark.parametrize("co", [HEAT, GENERAL, LIMIT], ids=["heat", "general", "limit"])
@pytest.mark.parametrize("n", PLACES)
@pytest.mark.parametrize("pad", [0, 1])
def test_contiguous(cuda, oracle, co, n, pad):
    """pad: systems n + pad apart, so that both parities of the distance are met."""
    k = 83
    d = np.random.default_rng(n).normal(size=(k, n + pad))
    t = torch.from_numpy(d).to(cuda)
    lay = (k, k, n + pad, 0, 1)
    want = oracle.exact_solve(np.ascontiguousarray(d[:, :n]), n, co)
    out = _solved(t, torch.full_like(t, 3.), n, co, lay, 2).cpu().numpy()
    old = _solved(t, torch.full_like(t, 3.), n, co, lay, 1).cpu().numpy()
    assert not np.array_equal(out, old)  # the forced kernel ran
    got = _solved(t, t, n, co, lay, 2).cpu().numpy()
    assert oracle.rel_err(out[:, :n], want) < TOL and (out[:, n:] == 3.).all()
    assert oracle.rel_err(got[:, :n], want) < TOL and np.array_equal(got[:, n:], d[:, n:])


@pytest.mark.parametrize("co", [HEAT, LIMIT], ids=["heat", "limit"])
@pytest.mark.parametrize("n", PLACES + [385, 512])
@pytest.mark.parametrize("planes,ni,es", [(1, 37, 38), (1, 37, 39), (9, 21, 21), (5, 7, 8)])
def test_strided(cuda, oracle, co, n, planes, ni, es):
    """es odd: no tensor maps.  Elements beyond a plane's systems stay."""
    if n == 512 and es % 2 == 0:
        pytest.skip("the 512-row kernels' own layout")
    d = np.random.default_rng(n).normal(size=(planes, n, es))
    t = torch.from_numpy(d).to(cuda)
    lay = (planes * ni, ni, 1, n * es, es)
    lines = np.moveaxis(d[:, :, :ni], 1, 2).reshape(-1, n)
    want = oracle.exact_solve(np.ascontiguousarray(lines), n, co)
    out = _solved(t, torch.full_like(t, 3.), n, co, lay, 2).cpu().numpy()
    old = _solved(t, torch.full_like(t, 3.), n, co, lay, 1).cpu().numpy()
    assert not np.array_equal(out, old)
    got = _solved(t, t, n, co, lay, 2).cpu().numpy()
    for o, rest in ((out, 3.), (got, d[:, :, ni:])):
        assert (o[:, :, ni:] == rest).all()
        assert oracle.rel_err(np.moveaxis(o[:, :, :ni], 1, 2).reshape(-1, n), want) < TOL


@pytest.mark.parametrize("n", PLACES)
@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("width", [18, 19])
def test_compact_derivative(cuda, oracle, n, axis, width):
    import ntk

    shape = [3, width, width]
    shape[axis] = n
    f = np.random.default_rng(n).normal(size=shape)
    ft = torch.from_numpy(f).to(cuda)
    out, old = torch.empty_like(ft), torch.empty_like(ft)
    h = 1. / (n - 1)
    with ntk.Plan(n, 0, COMPACT, precision="fp32_refine") as p:
        p.set_tuning(refine_kernel=1)
        p.compact_deriv(ft, old, axis, h)
        p.set_tuning(refine_kernel=2)
        p.compact_deriv(ft, out, axis, h)
        p.compact_deriv(ft, ft, axis, h)
        assert p.status() == 0
    assert not torch.equal(out, old)
    lines = np.ascontiguousarray(np.moveaxis(f, axis, 2)).reshape(-1, n)
    rhs = np.empty_like(lines)
    rhs[:, 1:-1] = 3 / (4 * h) * (lines[:, 2:] - lines[:, :-2])
    rhs[:, 0] = (-5 * lines[:, 0] + 4 * lines[:, 1] + lines[:, 2]) / (2 * h)
    rhs[:, -1] = (5 * lines[:, -1] - 4 * lines[:, -2] - lines[:, -3]) / (2 * h)
    want = oracle.exact_solve(rhs, n, COMPACT)
    for o in (out, ft):
        assert oracle.rel_err(np.moveaxis(o.cpu().numpy(), axis, 2).reshape(-1, n), want) < TOL


@pytest.mark.parametrize("n,few,many,strided", [(128, 2432, 16384, False), (97, 6001, 16384, False),
                                                (256, 2560, 16384, True), (385, 4867, 16385, True)])
def test_small_batches_keep_the_chunked_kernels(cuda, n, few, many, strided):
    for k, kernel in ((few, 1), (many, 2)):
        t = torch.from_numpy(np.random.default_rng(n).normal(size=(n, k) if strided else (k, n))).to(cuda)
        lay = (k, k, 1, 0, k) if strided else (k, k, n, 0, 1)
        by_rule, forced, other = (_solved(t, torch.empty_like(t), n, HEAT, lay, q) for q in (0, kernel, 3 - kernel))
        assert torch.equal(by_rule, forced) and not torch.equal(by_rule, other)
