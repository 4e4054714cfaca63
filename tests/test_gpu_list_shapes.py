"""Launch shapes and the autotuner where SSPRK steps run on neighbour lists,
whose passes choose their own shape (@gpu)."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import gpu_context, gpu_state

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
