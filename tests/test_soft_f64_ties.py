"""FP64 products on the integer pipes round ties to even, as IEEE products do:
the header compiled for the host, and diagonal systems, whose solution is one
product a row, through every FP64 kernel that scales its rows that way."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT

B = 2. / 3  # 1 / B is the double 1.5: one product in six is a tie


def test_ties_round_to_even(tmp_path):
    exe = tmp_path / "soft_f64_ties"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-I", cuda, "-o", str(exe),
                    os.path.join(ROOT, "tests", "soft_f64_ties.cpp")], check=True)
    res = subprocess.run([str(exe)], stdout=subprocess.PIPE, check=True).stdout
    checked, ties, wrong, untied, wrong_untied, wide, wrong_wide = map(int, res.split())
    assert checked > 4000000 and ties > 50000 and untied > 100000
    assert wrong == 0 and wrong_untied == 0
    assert wide > 500000 and wrong_wide == 0


# 3 systems: several threads a system; 300000: one thread a system
@pytest.mark.gpu
@pytest.mark.parametrize("nsys,n", [(3, 100), (300000, 40)])
@pytest.mark.parametrize("strided", [False, True])
def test_diagonal_solve_is_the_ieee_product(cuda, nsys, n, strided):
    import ntk
    import torch

    d = torch.from_numpy(np.random.default_rng(n).normal(size=(nsys, n))).to(cuda)
    want = d * (1. / B)
    with ntk.Plan(n, nsys, (B, 0., 0., B, 0., 0., B)) as p:
        if strided:
            t = d.t().contiguous()
            p.solve_strided(t, t, nsys, nsys, 1, 0, nsys)
            got = t.t()
        else:
            got = d.clone()
            p.solve(got)
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_diagonal_batch_is_the_ieee_product(cuda):
    import ntk
    import torch

    n = np.array([40, 700, 3000, 512, 17], dtype=np.int32)
    row = np.array([0., B, 0.])
    d = torch.from_numpy(np.random.default_rng(1).normal(size=int(n.sum()))).to(cuda)
    want = d * (1. / B)
    with ntk.UnevenBatch(n, np.tile(row, (5, 1)), np.tile(row, (5, 2, 1)), np.tile(row, (5, 2, 1))) as b:
        b.solve(d)
    assert torch.equal(d, want)
