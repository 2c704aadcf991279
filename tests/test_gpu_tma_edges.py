"""Strided batches whose rows are wider than their systems, an odd number of
them: tensor-map stores write 16-byte units, so the element behind the last
system of a row shares a unit with it.  It is neither written nor taken for an
input (whatever it holds, no range status), in FP32 and FP32 + refinement, by
every kernel that can serve the layout."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HEAT = (1., 0., -.5, 2., -.5, 0., 1.)


@pytest.mark.parametrize("precision,tol", [("fp32", 2e-5), ("fp32_refine", 1e-12)])
@pytest.mark.parametrize("kernel", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [385, 512, 700])
@pytest.mark.parametrize("planes,ni,es", [(1, 1, 6), (1, 7, 12), (3, 15, 16), (2, 33, 34), (1, 34, 36)])
@pytest.mark.parametrize("pad", [0.25, float("inf")])
def test_elements_beside_the_systems(cuda, oracle, precision, tol, kernel, n, planes, ni, es, pad):
    import ntk

    d = np.random.default_rng(n + ni).normal(size=(planes, n, es))
    d[:, :, ni:] = pad
    t = torch.from_numpy(d).to(cuda)
    out = torch.full_like(t, 3.)
    with ntk.Plan(n, 0, HEAT, precision=precision) as p:
        p.set_tuning(refine_kernel=kernel)
        p.solve_strided(t, out, planes * ni, ni, 1, n * es, es)
        p.solve_strided(t, t, planes * ni, ni, 1, n * es, es)
        assert p.status(raise_on_error=False) == 0
    lines = np.ascontiguousarray(np.moveaxis(d[:, :, :ni], 1, 2)).reshape(-1, n)
    want = oracle.exact_solve(lines, n, HEAT)
    for o, rest in ((out.cpu().numpy(), 3.), (t.cpu().numpy(), d[:, :, ni:])):
        assert (o[:, :, ni:] == rest).all()
        assert oracle.rel_err(np.moveaxis(o[:, :, :ni], 1, 2).reshape(-1, n), want) < tol
