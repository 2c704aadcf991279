"""Plans of different sizes used by several host threads at once, each on its
own stream: their launches share kernels but not shared-memory sizes.  A launch
that fails (its limit lowered by another thread's) raises."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HEAT = (1., 0., -.5, 2., -.5, 0., 1.)


def _in_threads(jobs):
    errors = []

    def run(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                job()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[:3]


@pytest.mark.parametrize("precision,sizes,nsys", [("fp64", (1024, 1500, 2048, 4096), 8),
                                                  ("fp32_refine", (100, 200, 400, 512), 31)])
def test_strided_solves_of_several_sizes(cuda, oracle, precision, sizes, nsys):
    jobs, checks = [], []
    import ntk

    for n in sizes:
        d = np.random.default_rng(n).normal(size=(nsys, n))
        t = torch.from_numpy(d.T.copy()).to(cuda)
        out = torch.empty_like(t)
        plan = ntk.Plan(n, 0, HEAT, precision=precision)

        def job(plan=plan, t=t, out=out):
            for _ in range(2000):
                plan.solve_strided(t, out, nsys, nsys, 1, 0, nsys)

        jobs.append(job)
        checks.append((plan, out, oracle.exact_solve(d, n, HEAT)))
    torch.cuda.synchronize()
    _in_threads(jobs)
    for plan, out, want in checks:
        assert oracle.rel_err(out.cpu().numpy().T, want) < 1e-12
        plan.close()


def test_adi_of_several_sizes(cuda):
    import ntk

    jobs = []
    for N in (200, 256, 999, 1100):
        dx = 1. / (N - 1)
        u = torch.randn((N, N), dtype=torch.float64, device=cuda)
        x, y = u.clone(), u.t().contiguous()
        a = ntk.Adi(N, dx, dx * dx)

        def job(a=a, u=u, x=x, y=y):
            for _ in range(500):
                a.step(u, x, y)

        jobs.append(job)
    torch.cuda.synchronize()
    _in_threads(jobs)
