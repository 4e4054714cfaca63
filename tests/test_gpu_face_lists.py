"""2D face walls finer than the particles: counts of segments within reach on
both sides of a face particle's list (@gpu)."""

from __future__ import annotations

import numpy as np
import pytest

from titsolver_gb300 import _abi, physics, scenarios

from helpers import fluid_mask, gpu_context, gpu_state, oracle_run, rel_l2

pytestmark = pytest.mark.gpu


def fine_pool(nx, finer):
    scn = scenarios.dam_break_2d_faces(nx_per_H=nx)
    n, H = scn["tanks"][0]["n_fluid"], scn["H"]
    walls, faces = scenarios.rectangle_faces(5.366 * H, 4.0 * H, scn["dx"] / finer)
    r = np.concatenate([scn["r"][:n], walls])
    rho = np.concatenate([scn["rho"][:n], np.full(len(walls), 1000.0)])
    return dict(scn, tanks=[dict(scn["tanks"][0], n_wall=len(walls))], r=r,
                v=np.zeros_like(r), rho=rho,
                faces=[dict(scn["faces"][0], face_verts=faces)])


# A particle one spacing from a wall has 7.7 spacings of it within reach (8 at
# the walls themselves): 61, 64, 69; 248, 256, 264 segments.
@pytest.mark.parametrize("finer", (8, 9, 32, 34))
def test_segments_around_the_list(gpu_lib, finer):
    scn = fine_pool(10, finer)
    P = physics.reference_params(2)
    P.post_integrate = _abi.TG_POST_SHIFTING
    o, f = oracle_run(scn, P, 1), fluid_mask(scn)
    with gpu_context(scn, P) as ctx:
        ctx.step(1)
        g = gpu_state(ctx)
    for key in ("r", "v", "rho"):
        assert rel_l2(g[key][f], getattr(o, key)[f]) <= 1e-11, key


@pytest.mark.parametrize("precision", (_abi.TG_FP64, _abi.TG_FP32C))
def test_dropped_faces_leave_the_steps(gpu_lib, precision):
    # Steps replay graphs: those with faces go with the faces.
    scn = scenarios.dam_break_2d_faces(nx_per_H=20)
    P = physics.reference_params(2, precision=precision)
    out = []
    for faces in (True, False):
        with gpu_context(scn if faces else dict(scn, faces=None), P) as ctx:
            if faces:
                ctx.step(5)
                ctx.set_faces(0, np.empty((0, 2)), np.empty((0, 2)))
            ctx.update(scn["r"], scn["v"], scn["rho"])
            ctx.step(5)
            out.append(gpu_state(ctx))
    for key in ("r", "v", "rho"):
        np.testing.assert_array_equal(out[0][key], out[1][key])
