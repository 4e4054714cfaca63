"""The roots and reciprocals of common.cuh against the host's long double, and
points so close that their squared distance is a subnormal number (@gpu)."""

from __future__ import annotations

import pathlib
import subprocess

import numpy as np
import pytest

import oracle
from helpers import fluid_mask, gpu_context, gpu_state, rel_l2
from titsolver_gb300 import _abi, build, physics, scenarios

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent

# Derived beside each function.  wall_density_f64: the roundings of y0^6 (5/6
# ulp of 2^-53 relative), of the last two operations and of e; FP32: the last
# rounding and the truncation.
BOUNDS = dict(rcp_f64=0.6, sqrt_f64=1.2, rcp_newton=0.51, sqrt_newton=0.51,
              wall_density_f64=2.0, sqrt_f64_tiny=0.0)


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


@pytest.mark.parametrize("kernel", (_abi.TG_KERNEL_WENDLAND_C2, _abi.TG_KERNEL_CUBIC_SPLINE))
def test_density_of_nearly_coincident_points(gpu_lib, kernel):
    r = np.zeros((40, 3))
    r[1, 0], r[2, 1], r[3, 2] = 1e-155, 3e-156, -2e-158
    r[4:] = np.random.default_rng(4).uniform(-0.2, 0.2, (36, 3))
    scn = dict(dim=3, tanks=[dict(n_fluid=40, n_wall=0, h=0.1, m=0.5, rho0=1000.0, cs0=1.0)],
               r=r, v=np.zeros_like(r), rho=np.full(40, 1000.0))
    with gpu_context(scn, physics.baseline_params(3, kernel=kernel)) as ctx:
        rho, cnt, _ = ctx.summation_density(_abi.TG_POS_FP64)
    o = oracle.summation_density(r, 0.1, 0.5, kernel, _abi.TG_POS_FP64)
    np.testing.assert_array_equal(cnt, o[1])
    np.testing.assert_allclose(rho, o[0], rtol=1e-12)


def test_step_with_nearly_coincident_particles(gpu_lib):
    # Two particles with a subnormal squared distance step as coincident ones
    # do (their pair adds nothing until they have parted), and with the terms
    # that divide by the distance their state stays finite.
    scn = scenarios.dam_break_2d(nx_per_H=10)
    out = []
    for gap in (0.0, 1e-155):
        r = scn["r"] - scn["r"][95]
        r[95] = 0.0
        r[96] = (gap, 0.0)
        with gpu_context(dict(scn, r=r), physics.baseline_params(2)) as ctx:
            ctx.step(1)
            out.append(gpu_state(ctx))
    f = fluid_mask(scn)
    for key in ("r", "v", "rho"):
        assert rel_l2(out[1][key][f], out[0][key][f]) <= 1e-12, key
    with gpu_context(dict(scn, r=r), physics.reference_params(2)) as ctx:
        ctx.step(1)
        assert np.all(np.isfinite(gpu_state(ctx)["v"]))
