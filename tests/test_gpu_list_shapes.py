"""Launch shapes and the autotuner where SSPRK steps run on neighbour lists,
whose passes choose their own shape (@gpu)."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import fluid_mask, gpu_context, gpu_state, oracle_run, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", (_abi.TG_FP64, _abi.TG_FP32C))
def test_list_steps_do_not_depend_on_the_shape(gpu_lib, precision):
    # 20,000 particles: one lane each, and no chains in the plain form.
    scn = scenarios.dam_break_2d(nx_per_H=100)
    out = []
    for block, lanes in ((128, 1), (64, 4), (256, 2)):
        with gpu_context(scn, physics.baseline_params(2, precision=precision)) as ctx:
            ctx.set_tuning(2, block, lanes)
            ctx.step(4)
            out.append(gpu_state(ctx))
    for other in out[1:]:
        for k in ("r", "v", "rho", "dv_dt", "drho_dt", "time"):
            np.testing.assert_array_equal(other[k], out[0][k], err_msg=k)


@pytest.mark.parametrize("precision", (_abi.TG_FP64, _abi.TG_FP32C))
def test_autotune_times_the_steps_alone(gpu_lib, precision):
    # No graph capture within the trials: their time per step is that of the
    # steps that follow (about .1 ms here, a capture takes over 1 ms).
    scn = scenarios.dam_break_2d(nx_per_H=20)
    with gpu_context(scn, physics.baseline_params(2, precision=precision)) as ctx:
        t = ctx.autotune(2)
        ctx.step(10)
        ctx.timer_start()
        ctx.step(50)
        ms = ctx.timer_stop() / 50
    assert t["ms_per_step"] <= 2.0 * ms
    # Cell sizes, then the walk's shapes: itself, lanes, blocks.
    assert t["candidates"] == 8


@pytest.mark.parametrize("integrator", (_abi.TG_SSPRK3, _abi.TG_EULER))
@pytest.mark.parametrize("xi,eos", ((5.0, _abi.TG_EOS_TAIT), (7.0, _abi.TG_EOS_LINEAR_TAIT)))
@pytest.mark.parametrize("term_set", ("baseline", "reference"))
@pytest.mark.parametrize("dim", (2, 3))
def test_presets_with_other_equations_of_state(gpu_lib, dim, term_set, xi, eos, integrator):
    # The compile-time terms, on lists and on the cell walk (bounds of the
    # compensated form after 30 steps).
    scn = (scenarios.dam_break_2d(nx_per_H=20) if dim == 2
           else scenarios.dam_break_3d(nx_per_H=8))
    P = getattr(physics, f"{term_set}_params")(dim)
    P.xi, P.eos, P.integrator = xi, eos, integrator
    o, f = oracle_run(scn, P, 5), fluid_mask(scn)
    P.precision = _abi.TG_FP32C
    with gpu_context(scn, P) as ctx:
        ctx.step(5)
        g = gpu_state(ctx)
    assert rel_l2(g["r"][f], o.r[f]) <= 1e-6
    assert rel_l2(g["rho"][f], o.rho[f]) <= 1e-5
