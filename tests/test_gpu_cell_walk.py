"""SSPRK steps that walk cells (a sort per stage), which stopped steps and
particle sets without room for neighbour lists take: terms, kernels, launch
shapes, staging, re-sort, shifting and face walls, against the oracle (@gpu).

A second tank of two walls 50,000 support radii apart, whose FP32 coordinates
do not resolve its radius, keeps a context off lists; bounds as in
test_gpu_step.py and test_gpu_tuning.py."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import fluid_mask, gpu_context, gpu_state, oracle_run, rel_l2

pytestmark = pytest.mark.gpu


def _walking(scn):
    far = np.zeros((2, scn["dim"]))
    far[1, 0] = 1e5
    tank = dict(scn["tanks"][0], n_fluid=0, n_wall=2, h=1.0)
    out = dict(scn, tanks=[*scn["tanks"], tank], r=np.concatenate([scn["r"], far]),
               v=np.concatenate([scn["v"], 0.0 * far]),
               rho=np.concatenate([scn["rho"], [tank["rho0"]] * 2]))
    if scn.get("faces"):
        out["faces"] = [*scn["faces"], None]
    return out


def _steps(scn, P, steps, shape=None):
    with gpu_context(_walking(scn), P) as ctx:
        if shape is not None:
            ctx.set_tuning(*shape)
        before = ctx.launch_count()
        ctx.step(steps)
        assert ctx.launch_count() - before > 40 * steps  # about 20 on lists
        g = gpu_state(ctx)
    n = scn["r"].shape[0]
    return {k: a[:n] for k, a in g.items()}


def _check(scn, P64, steps, precision, shape=None, state=1e-12, deriv=1e-9):
    o, f = oracle_run(scn, P64, steps), fluid_mask(scn)
    P = _abi.TgParams.from_buffer_copy(P64)
    P.precision = precision
    g = _steps(scn, P, steps, shape)
    if precision == _abi.TG_FP64:
        assert rel_l2(g["r"][f], o.r[f]) <= state
        assert rel_l2(g["rho"][f], o.rho[f]) <= state
        assert rel_l2(g["dv_dt"][f], o.dv_dt[f]) <= deriv
    else:
        assert rel_l2(g["r"][f], o.r[f]) <= 1e-6
        assert rel_l2(g["rho"][f], o.rho[f]) <= 1e-5


@pytest.mark.parametrize("term_set", ("baseline", "reference"))
@pytest.mark.parametrize("lanes", (1, 2, 4))
@pytest.mark.parametrize("k,block", ((1, 128), (2, 64), (3, 256)))
def test_walk_shapes_2d(gpu_lib, term_set, lanes, k, block):
    scn = scenarios.dam_break_2d(nx_per_H=20)
    P = getattr(physics, f"{term_set}_params")(2)
    _check(scn, P, 2, _abi.TG_FP64, (k, block, lanes))
    _check(scn, P, 30, _abi.TG_FP32C, (k, block, lanes))


@pytest.mark.parametrize("shape", ((1, 128, 4), (2, 256, 2), (3, 64, 1)))
def test_walk_shapes_3d(gpu_lib, shape):
    scn, P = scenarios.dam_break_3d(nx_per_H=8), physics.baseline_params(3)
    _check(scn, P, 1, _abi.TG_FP64, shape)
    _check(scn, P, 10, _abi.TG_FP32C, shape)


@pytest.mark.parametrize("kernel", range(6))
@pytest.mark.parametrize("dim", (2, 3))
def test_walk_kernels(gpu_lib, dim, kernel):
    scn = (scenarios.dam_break_2d(nx_per_H=10) if dim == 2
           else scenarios.dam_break_3d(nx_per_H=7))
    P = physics.reference_params(dim, kernel=kernel)
    _check(scn, P, 1, _abi.TG_FP64)
    _check(scn, P, 5, _abi.TG_FP32C)


@pytest.mark.parametrize("xi,eos,kahan", ((5.0, _abi.TG_EOS_TAIT, 1),
                                          (7.0, _abi.TG_EOS_LINEAR_TAIT, 1),
                                          (7.0, _abi.TG_EOS_TAIT, 0)))
def test_walk_generic_terms(gpu_lib, xi, eos, kahan):
    scn, P = scenarios.dam_break_2d(nx_per_H=20), physics.baseline_params(2)
    P.xi, P.eos, P.kahan = xi, eos, kahan
    _check(scn, P, 2, _abi.TG_FP64)
    _check(scn, P, 10, _abi.TG_FP32C)


@pytest.mark.parametrize("precision", (_abi.TG_FP64, _abi.TG_FP32C))
@pytest.mark.parametrize("case", ("2d", "3d", "faces"))
def test_walk_shifting(gpu_lib, case, precision):
    scn = (scenarios.dam_break_3d(nx_per_H=8) if case == "3d" else
           scenarios.dam_break_2d_faces(nx_per_H=20) if case == "faces" else
           scenarios.dam_break_2d(nx_per_H=20))
    P = physics.reference_params(scn["dim"])
    P.post_integrate = _abi.TG_POST_SHIFTING
    _check(scn, P, 2, precision, state=1e-11, deriv=1e-8)


@pytest.mark.parametrize("switch", ("staging", "resort"))
def test_walk_switches_bit_identical(gpu_lib, switch):
    # Staging visits the same candidates in the same order, and the re-sort
    # gives the full sort's order.
    scn = scenarios.dam_break_2d(nx_per_H=40)
    out = []
    for value in (1, 0):
        P = physics.baseline_params(2, precision=_abi.TG_FP32C)
        setattr(P, switch, value)
        out.append(_steps(scn, P, 5))
    for k in ("r", "v", "rho", "dv_dt", "drho_dt"):
        np.testing.assert_array_equal(out[0][k], out[1][k])
