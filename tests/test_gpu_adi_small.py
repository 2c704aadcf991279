"""FP64 ADI steps on both sides of the smallest grid that whole systems in
shared memory serve (N = 40), with and without a zero stencil centre and with
coefficients far from one.  Tolerance as in test_gpu_adi."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("N", [39, 40, 41, 79, 80])
@pytest.mark.parametrize("ratio", [1.0, 0.5, 80.0])
@pytest.mark.parametrize("length", [1., 1e-9])
def test_step_matches_the_oracle(cuda, oracle, N, ratio, length):
    import ntk

    dx = length / (N - 1)
    dt = ratio * dx * dx
    u = np.random.default_rng(N).normal(size=(N, N))
    u[:, : N // 2] = 0.  # a quiet region
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
