"""The FP32 form's quotient against correctly rounded division, with the bound its
three roundings give: tests/cuda/quotient_check.cu, built here for sm_100a and run
over 4.3e9 random quotients."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def build_and_run(name, tmp_path, *link):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / name)
    src = os.path.join(ROOT, "tests", "cuda", name + ".cu")
    inc = os.path.join(ROOT, "jenhine_b200", "csrc")
    b = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                        "-I", inc, src, *link, "-o", exe], capture_output=True, text=True, timeout=300)
    assert b.returncode == 0, b.stdout + b.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_quotients_are_correctly_rounded_but_near_a_middle(tmp_path):
    out = build_and_run("quotient_check", tmp_path)
    print(out)
    assert out.count(" 0 outside the bound, 0 forms disagree") == 2
