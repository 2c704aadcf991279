"""FP64 ADI steps at sizes on both sides of the choice between whole systems,
windows and segmented sweeps, with and without a zero stencil centre
(dt = dx^2) and with slowly decaying factors.  Tolerance as in test_gpu_adi."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("N", [4, 19, 20, 21, 100, 127, 128, 255, 401, 513, 700])
@pytest.mark.parametrize("ratio", [1.0, 0.5, 80.0])
def test_step_matches_the_oracle(cuda, oracle, N, ratio):
    import ntk

    dx = 1.0 / (N - 1)
    dt = ratio * dx * dx
    u = np.random.default_rng(N).normal(size=(N, N))
    want = u.copy()
    wdx, wdy = u.copy(), u.T.copy()
    for _ in range(2):
        oracle.adi_step_exact(want, wdx, wdy, dx, dt)
    ut = torch.from_numpy(u).to(cuda)
    d_x, d_y = ut.clone(), ut.t().contiguous()
    with ntk.Adi(N, dx, dt) as a:
        a.run(ut, d_x, d_y, 2, graph=(N % 2 == 0))
    assert oracle.rel_err(ut.cpu().numpy(), want) < TOL
    assert oracle.rel_err(d_x.cpu().numpy()[1:-1], wdx[1:-1]) < TOL
