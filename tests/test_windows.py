"""Overlapping windows with a halo longer than their central rows (slow decay):
none reaches outside its system.  The rule on the host (csrc/ntk_windows.h), and
the solves that use it on arrays inside buffers of nan, which any value read
beside the arrays would bring into the results."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT


def test_windows_stay_inside_the_system(tmp_path):
    exe = tmp_path / "windows_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "windows_check.cpp")], check=True)
    layouts, long_halos, wrong = map(int, subprocess.run([str(exe)], stdout=subprocess.PIPE, check=True).stdout.split())
    assert layouts > 50000 and long_halos > 1000
    assert wrong == 0


def _guarded(x):
    """x on the device inside a buffer of nan, 512 rows of it before and behind."""
    import torch

    g = 512 * x.shape[-1]
    buf = torch.full((x.size + 2 * g,), float("nan"), dtype=torch.float64, device="cuda")
    t = buf[g:g + x.size].view(x.shape)
    t.copy_(torch.from_numpy(np.ascontiguousarray(x)))
    return t


# ratio 2: halo 44 - 48 of 128-row windows; 8: 86 - 96 of 256; 30: of 512.  FP32 +
# refinement keeps 47 bits; a half step's matrix has condition 2 ratio + 1, which
# bounds its own error and what it makes of the half step before.
@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("fp32_refine", None), ("fp32", 1e-3)])
@pytest.mark.parametrize("N,ratio", [(129, 2.), (200, 2.), (255, 2.), (255, 1.9), (257, 8.), (400, 8.), (511, 7.),
                                     (513, 30.), (600, 30.), (1100, 28.), (1100, 40.)])
def test_adi(cuda, oracle, precision, tol, N, ratio):
    import ntk
    import torch

    if tol is None:
        tol = max(1e-12, 2. ** -47 * (2. * ratio + 1.) ** 2)
    dx = 1. / (N - 1)
    u = np.random.default_rng(N).normal(size=(N, N))
    want = u.copy()
    wx, wy = u.copy(), u.T.copy()
    oracle.adi_step_exact(want, wx, wy, dx, ratio * dx * dx)
    ut, x, y = _guarded(u), _guarded(u), _guarded(u.T)
    try:
        a = ntk.Adi(N, dx, ratio * dx * dx, precision=precision)
    except ntk.NtkError:
        pytest.skip("refused: decays too slowly for the windows")
    a.step(ut, x, y)
    torch.cuda.synchronize()
    assert a.status(raise_on_error=False) == 0
    a.close()
    assert oracle.rel_err(ut.cpu().numpy(), want) < tol


# multipliers 0.78 .. 0.814: halos of 158 to 190 rows of 512.  One FP32 solve is
# off by 2^-24 times the condition 1 + 4 r at most, a sweep squares that: 3.1e-11.
@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp32_refine", 3.1e-11), ("fp32", 1e-3)])
@pytest.mark.parametrize("r", [16., 18., 20., 23.])
@pytest.mark.parametrize("n", [700, 1025, 1300, 2500])
@pytest.mark.parametrize("strided", [False, True])
def test_long_systems(cuda, oracle, precision, tol, r, n, strided):
    import ntk
    import torch

    co = (1., 0., -r, 1. + 2. * r, -r, 0., 1.)
    k = 7
    d = np.random.default_rng(n).normal(size=(k, n))
    want = oracle.exact_solve(d, n, co)
    t = _guarded(d.T if strided else d)
    out = torch.empty_like(t)
    with ntk.Plan(n, 0, co, precision=precision) as p:
        p.set_tuning(refine_kernel=1, refine_tps=64)
        if strided:
            p.solve_strided(t, out, k, k, 1, 0, k)
        else:
            p.solve_strided(t, out, k, k, n, 0, 1)
        assert p.status(raise_on_error=False) == 0
    got = out.cpu().numpy().T if strided else out.cpu().numpy()
    assert oracle.rel_err(got, want) < tol
