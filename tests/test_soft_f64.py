"""The FP64 product on the integer pipes (csrc/ntk_soft_f64.cuh), the
product's own header compiled for the host: equal to the IEEE product for
every operand it takes (a result within 2^-62 of a rounding boundary could
differ; none of these is), and zeros, subnormals, infinities, NaNs and factors
beyond 2^+-60 are left to the FP64 pipe."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_soft_product_is_the_ieee_product(tmp_path):
    exe = tmp_path / "soft_f64_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-I", cuda, "-o", str(exe),
                    os.path.join(ROOT, "tests", "soft_f64_check.cpp")], check=True)
    checked, wrong, refused = map(int, subprocess.run([str(exe)], stdout=subprocess.PIPE, check=True).stdout.split())
    assert wrong == 0
    assert checked > 2000000 and refused > 100000
