"""The roots and reciprocals of common.cuh against the host's long double
(@gpu)."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

from titsolver_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent

# Derived beside each function.  wall_density_f64: the roundings of y0^6 (5/6
# ulp of 2^-53 relative), of the last two operations and of e; FP32: the last
# rounding and the truncation.
BOUNDS = dict(rcp_f64=0.6, sqrt_f64=1.2, rcp_newton=0.51, sqrt_newton=0.51,
              wall_density_f64=2.0)


def test_roots(tmp_path):
    exe = tmp_path / "roots"
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++20", "--extended-lambda",
                    "--expt-relaxed-constexpr", "-I", str(ROOT / "include"),
                    "-I", str(build.CSRC), str(ROOT / "tests" / "cpp" / "roots.cu"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    worst = {name: float(v) for name, v in (line.split() for line in out.splitlines())}
    assert worst.keys() == BOUNDS.keys()
    for name, bound in BOUNDS.items():
        assert worst[name] <= bound, (name, worst[name])
