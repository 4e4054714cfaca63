"""Steps that cannot be finished on their neighbour lists: what such a stop
leaves, what it costs, and the steps after it, against the oracle (@gpu)."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import fluid_mask, gpu_context, gpu_state, oracle_run, rel_l2

pytestmark = pytest.mark.gpu

# Relative L2 bounds of r, v, rho: ten times those of two steps in the plain
# form (ten steps here), those of 30 steps in the compensated form.
FORMS = ((_abi.TG_FP64, (1e-11, 1e-10, 1e-11)), (_abi.TG_FP32C, (1e-6, 1e-4, 1e-5)))


def _same(ctx, scn, o, tol):
    g, f = gpu_state(ctx), fluid_mask(scn)
    for key, bound in zip(("r", "v", "rho"), tol):
        assert rel_l2(g[key][f], getattr(o, key)[f]) <= bound, key
    np.testing.assert_allclose(g["time"], o.time, rtol=2e-6)


def _launches(ctx, steps):
    before = ctx.launch_count()
    ctx.step(steps)
    return ctx.launch_count() - before


def _closing_in(dim, faces, cfl):
    """Fluid that runs together at ten times the speed of sound: its lists
    outgrow their capacity after some steps."""
    scn = (scenarios.dam_break_3d(nx_per_H=8) if dim == 3 else
           scenarios.dam_break_2d_faces(nx_per_H=20) if faces else
           scenarios.dam_break_2d(nx_per_H=20))
    f = fluid_mask(scn)
    d = scn["r"][f] - scn["r"][f].mean(axis=0)
    v = np.zeros_like(scn["r"])
    v[f] = -d / np.linalg.norm(d, axis=1).max()
    rho = np.full(f.size, 1000.0)
    P = physics.baseline_params(dim)
    P.cfl = cfl
    P.g = 1e-3
    return dict(scn, v=v, rho=rho, tanks=[dict(scn["tanks"][0], cs0=0.1)]), P


# In chains (the capacity ends one after the first), with shifting and with
# face walls (steps one by one); the plain form of these sizes chains as well.
@pytest.mark.parametrize("dim,faces,shifting,cfl,steps",
                         ((2, False, False, 0.15, 8), (3, False, False, 0.08, 8),
                          (2, False, True, 0.2, 12), (3, False, True, 0.11, 10),
                          (2, True, False, 0.2, 12), (2, True, True, 0.2, 12)))
def test_stop_after_finished_steps(gpu_lib, dim, faces, shifting, cfl, steps):
    scn, P64 = _closing_in(dim, faces, cfl)
    if shifting:
        P64.post_integrate = _abi.TG_POST_SHIFTING
    o = oracle_run(scn, P64, steps)
    for precision, tol in FORMS:
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        with gpu_context(scn, P) as ctx:  # as the stop's first half: no stop yet
            first = _launches(ctx, 2)
        with gpu_context(scn, P) as ctx:
            # One step of the cell walk takes over 45 launches more.
            assert _launches(ctx, steps) > steps // 2 * first + 45
            _same(ctx, scn, o, tol)


@pytest.mark.parametrize("dim", (2, 3))
def test_stop_in_the_second_step_of_a_chain(gpu_lib, dim):
    # Free fall from rest: the chain's bound is its margin alone, which the
    # first step keeps and the second one does not.  Single steps do not stop.
    scn = (scenarios.dam_break_2d(nx_per_H=20, hydrostatic=False) if dim == 2
           else scenarios.dam_break_3d(nx_per_H=8))
    scn = dict(scn, rho=np.full(scn["rho"].size, 1000.0),
               tanks=[dict(scn["tanks"][0], cs0=1.0)])
    P64 = physics.baseline_params(dim)
    P64.c_force = 0.167
    for precision, tol in FORMS:
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        o = oracle_run(scn, P64, 2)
        with gpu_context(scn, P) as ctx:
            single = _launches(ctx, 1) + _launches(ctx, 1)
            assert single <= 90
            _same(ctx, scn, o, tol)
        with gpu_context(scn, P) as ctx:
            assert _launches(ctx, 2) > single + 30
            _same(ctx, scn, o, tol)
            # The next call is back on lists, one step at a time.
            assert _launches(ctx, 2) <= 90
            _same(ctx, scn, oracle_run(scn, P64, 4), tol)


def test_stop_in_the_post_integration_stage(gpu_lib):
    # As above with shifting: the first step's end is beyond the bound.
    scn = scenarios.dam_break_2d(nx_per_H=20, hydrostatic=False)
    scn = dict(scn, tanks=[dict(scn["tanks"][0], cs0=1.0)])
    P64 = physics.baseline_params(2)
    P64.c_force = 0.167
    P64.post_integrate = _abi.TG_POST_SHIFTING
    for precision, tol in FORMS:
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        with gpu_context(scn, P) as ctx:
            # A step with shifting takes about 30 launches on lists.
            assert _launches(ctx, 1) > 75
            _same(ctx, scn, oracle_run(scn, P64, 1), tol)
            assert _launches(ctx, 2) <= 75
            _same(ctx, scn, oracle_run(scn, P64, 3), tol)


def _bursting(nx):
    # A block at half more than the reference density: its first steps throw
    # the particles around it far beyond the bound.
    scn = scenarios.dam_break_2d(nx_per_H=nx)
    rho = scn["rho"].copy()
    n = scn["tanks"][0]["n_fluid"]
    r = scn["r"][:n]
    rho[:n][np.abs(r - np.array([1.0, 0.5])).max(axis=1) < 0.08] = 1500.0
    return dict(scn, rho=rho)


def test_long_call_goes_back_to_lists(gpu_lib):
    # A stop costs a few steps, not the rest of the call: a walked step takes
    # over 45 launches more than one on lists (about 30).
    scn = _bursting(20)
    P64 = physics.baseline_params(2)
    P64.cfl = 1.0
    for precision, tol in FORMS:
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        with gpu_context(scn, P) as ctx:
            assert _launches(ctx, 3) > 135
            _same(ctx, scn, oracle_run(scn, P64, 3), tol)
        with gpu_context(scn, P) as ctx:
            assert _launches(ctx, 400) < 45 * 400
            calm = [_launches(ctx, 20) for _ in range(5)]
            assert max(calm) <= 45 * 20


def test_stops_in_every_call(gpu_lib):
    # Six calls whose start states each stop their lists.
    scn = _bursting(20)
    P64 = physics.baseline_params(2)
    P64.cfl = P64.c_force = 4.0
    P = _abi.TgParams.from_buffer_copy(P64)
    o = oracle_run(scn, P64, 1)
    f = fluid_mask(scn)
    with gpu_context(scn, P) as ctx:
        for _ in range(6):
            ctx.update(scn["r"], scn["v"], scn["rho"])
            ctx.step(1)
            g = gpu_state(ctx)
            assert rel_l2(g["r"][f], o.r[f]) <= 1e-12
            assert rel_l2(g["rho"][f], o.rho[f]) <= 1e-12
