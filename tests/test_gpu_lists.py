"""Steps on neighbour lists: every width of the list passes, steps that have
to be repeated with a sort per stage, and particles outside the grid, against
the oracle (@gpu)."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import fluid_mask, gpu_context, gpu_state, oracle_run, rel_l2

pytestmark = pytest.mark.gpu


def _check(scn, P64, steps, move=None, repeated=False):
    """Both forms against the oracle's FP64 run; move(r) edits the positions
    after the upload (whose positions make the grid).  repeated: the steps
    are expected to be repeated with a sort per stage (many more launches)."""
    r = scn["r"].copy()
    if move is not None:
        move(r)
    o = oracle_run(dict(scn, r=r), P64, steps)
    f = fluid_mask(scn)
    for precision, tol_r, tol_v, tol_rho in ((_abi.TG_FP64, 1e-12, 1e-11, 1e-12),
                                             (_abi.TG_FP32C, 1e-6, 1e-4, 1e-5)):
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        with gpu_context(scn, P) as ctx:
            if move is not None:
                ctx.update(r, scn["v"], scn["rho"])
            before = ctx.launch_count()
            ctx.step(steps)
            assert (ctx.launch_count() - before > 45 * steps) == repeated
            g = gpu_state(ctx)
        assert rel_l2(g["r"][f], o.r[f]) <= tol_r
        assert rel_l2(g["v"][f], o.v[f]) <= tol_v
        assert rel_l2(g["rho"][f], o.rho[f]) <= tol_rho


def _jittered(scn, amount=0.1, seed=3):
    rng = np.random.default_rng(seed)
    f = fluid_mask(scn)
    r = scn["r"].copy()
    r[f] += rng.uniform(-amount, amount, r[f].shape) * scn["dx"]
    return dict(scn, r=r)


# 16, 4 and 1 lanes per particle: fluid counts on both sides of the limits
# (32 and 128 particles per multiprocessor; 152 of them).
@pytest.mark.parametrize("dim,nx", ((2, 11), (2, 49), (2, 50), (2, 98), (2, 99), (2, 199), (3, 9),
                                    (3, 15), (3, 23)))
def test_list_widths(gpu_lib, dim, nx):
    scn = (scenarios.dam_break_2d(nx_per_H=nx) if dim == 2
           else scenarios.dam_break_3d(nx_per_H=nx, column=(1.7, 1.0, 1.0)))
    _check(_jittered(scn), physics.baseline_params(dim), 2)


@pytest.mark.parametrize("dim,nx", ((2, 11), (2, 50), (2, 98), (2, 99), (3, 9), (3, 15), (3, 23)))
def test_shifting_on_lists(gpu_lib, dim, nx):
    # The post-integration passes at the same widths.
    scn = _jittered(scenarios.dam_break_2d(nx_per_H=nx) if dim == 2 else
                    scenarios.dam_break_3d(nx_per_H=nx, column=(1.7, 1.0, 1.0)))
    P64 = physics.baseline_params(dim)
    P64.post_integrate = _abi.TG_POST_SHIFTING
    o = oracle_run(scn, P64, 2)
    f = fluid_mask(scn)
    # FP64: the bound of the existing 2-step shifting tests; compensated form:
    # theirs after 30 steps.
    for precision, tol_r, tol_v, tol_rho in ((_abi.TG_FP64, 1e-11, 1e-11, 1e-11),
                                             (_abi.TG_FP32C, 1e-6, 1e-4, 1e-5)):
        P = _abi.TgParams.from_buffer_copy(P64)
        P.precision = precision
        with gpu_context(scn, P) as ctx:
            ctx.step(1)
            ctx.step(1)
            g = gpu_state(ctx)
        assert rel_l2(g["r"][f], o.r[f]) <= tol_r
        assert rel_l2(g["v"][f], o.v[f]) <= tol_v
        assert rel_l2(g["rho"][f], o.rho[f]) <= tol_rho


@pytest.mark.parametrize("kernel", range(6))
def test_list_kernels_and_generic_terms(gpu_lib, kernel):
    # Every kernel's list sums, with terms that no compile-time preset covers
    # (Monaghan viscosity beside Ferrari diffusion, xi = 5).
    P = physics.baseline_params(3, kernel=kernel)
    P.diffusion = _abi.TG_DIFF_FERRARI
    P.xi = 5.0
    _check(_jittered(scenarios.dam_break_3d(nx_per_H=7)), P, 2)


@pytest.mark.parametrize("dim", (2, 3))
def test_steps_beyond_the_displacement_bound_are_repeated(gpu_lib, dim):
    # A CFL number of 4 and a density bump: the accelerations of the first
    # stage move particles past the bound that the lists were built for.
    scn = (scenarios.dam_break_2d(nx_per_H=20) if dim == 2
           else scenarios.dam_break_3d(nx_per_H=8))
    rho = scn["rho"].copy()
    rho[:: 7][: scn["tanks"][0]["n_fluid"] // 7] *= 1.08
    P = physics.baseline_params(dim)
    P.cfl = 4.0
    P.c_force = 4.0
    _check(dict(scn, rho=rho), P, 2, repeated=True)


def test_lists_past_their_capacity_are_repeated(gpu_lib):
    # Four times the mass for the spacing: a quarter of the neighbours that
    # the lists make room for.
    scn = scenarios.dam_break_2d(nx_per_H=20)
    tanks = [dict(scn["tanks"][0], m=4.0 * scn["tanks"][0]["m"])]
    _check(dict(scn, tanks=tanks), physics.baseline_params(2), 3, repeated=True)


@pytest.mark.parametrize("dim", (2, 3))
def test_particles_outside_the_grid(gpu_lib, dim):
    # A lump of fluid far above the grid, and another one across its border.
    scn = _jittered(scenarios.dam_break_2d(nx_per_H=20) if dim == 2
                    else scenarios.dam_break_3d(nx_per_H=8))
    lo, hi = scn["r"][:, 1].min(), scn["r"][:, 1].max()
    n = scn["tanks"][0]["n_fluid"]

    def move(r):
        r[: n // 8, 1] += 2.0 * (hi - lo)
        r[n // 8: n // 4, 1] += 1.3 * (hi - lo)

    _check(scn, physics.baseline_params(dim), 2, move)


@pytest.mark.parametrize("dim", (2, 3))
@pytest.mark.parametrize("steps", (1, 2, 3, 5))
def test_chained_steps(gpu_lib, dim, steps):
    # The compensated form's steps share their lists in pairs; tanks of
    # different time steps, odd counts, and the time of every tank.
    scn = (scenarios.batched_tanks(n_tanks=4, n_range=(8, 21), seed=7) if dim == 2
           else scenarios.batched_tanks_3d(n_tanks=3, n_range=(5, 9), seed=7))
    scn = _jittered(scn)
    P = physics.baseline_params(dim)
    _check(scn, P, steps)
    o = oracle_run(scn, P, steps)
    P.precision = _abi.TG_FP32C
    with gpu_context(scn, P) as ctx:
        dt = ctx.step(steps)
        np.testing.assert_allclose(ctx.time(), o.time, rtol=2e-6)
        np.testing.assert_allclose(dt, o.dt, rtol=2e-6)
