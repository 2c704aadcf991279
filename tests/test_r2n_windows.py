"""The windows of the paired-chunk solve of any length (csrc/ntk_r2n_windows.h,
compiled for the host), over lengths, halos and both group sizes."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_accepted_windows_cover_every_row_once(tmp_path):
    exe = tmp_path / "r2n_windows_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "r2n_windows_check.cpp")], check=True)
    layouts, accepted, wrong = map(int, subprocess.run([str(exe)], stdout=subprocess.PIPE, check=True).stdout.split())
    assert layouts > 300000 and accepted > .9 * layouts
    assert wrong == 0
