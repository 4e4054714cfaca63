"""Summation density of point clouds at the edges of its kernels: counts
around a warp, more neighbours than a warp's queue holds, coincident points,
every kernel, both position precisions, and the entry point that allocates
nothing, against the oracle (@gpu)."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle
from helpers import gpu_context
from titsolver_gb300 import _abi, physics

pytestmark = pytest.mark.gpu


def _cloud(n, dim, centre):
    rng = np.random.default_rng(n + 10 * dim)
    r = centre + rng.uniform(0.0, 1.0, (n, dim))
    r[n // 2: n // 2 + n // 8] = r[: n // 8]  # coincident points
    r[-1] = centre + 5.0                      # one far from all others
    return np.ascontiguousarray(r)


def _check(rho, cnt, hs, o, tol):
    np.testing.assert_array_equal(cnt, o[1])
    np.testing.assert_array_equal(hs, o[2])
    np.testing.assert_allclose(rho, o[0], rtol=tol)


# FP64: the order of at most ~1000 positive terms (1e-13); FP32: the oracle
# sums that many plainly in FP32 (1000 x 2^-24 at worst, 6e-5 / 6).
@pytest.mark.parametrize("dim", (2, 3))
@pytest.mark.parametrize("n", (1, 2, 31, 33, 1025))
def test_density_sizes(gpu_lib, dim, n):
    torch = pytest.importorskip("torch")
    h, m = 0.15, 0.5
    for centre in (0.0, -37.25):
        r = _cloud(n, dim, centre)
        scn = dict(dim=dim, tanks=[dict(n_fluid=n, n_wall=0, h=h, m=m, rho0=1000.0, cs0=1.0)],
                   r=r, v=np.zeros_like(r), rho=np.full(n, 1000.0))
        with gpu_context(scn, physics.baseline_params(dim)) as ctx:
            for precision, tol in ((_abi.TG_POS_FP64, 1e-12), (_abi.TG_POS_FP32, 1e-5)):
                o = oracle.summation_density(r, h, m, _abi.TG_KERNEL_WENDLAND_C2, precision)
                _check(*ctx.summation_density(precision), o, tol)
        r_d = torch.from_numpy(r).cuda()
        rho = torch.empty(n, dtype=torch.float64, device="cuda")
        cnt = torch.empty(n, dtype=torch.int32, device="cuda")
        hs = torch.empty(n, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        st = gpu_lib.tg_summation_density_noalloc(
            dim, _abi.TG_KERNEL_WENDLAND_C2, n, ctypes.c_void_p(r_d.data_ptr()), h, m,
            *(ctypes.c_void_p(a.data_ptr()) for a in (rho, cnt, hs)), None)
        torch.cuda.synchronize()
        assert st == _abi.TG_OK
        o = oracle.summation_density(r, h, m, _abi.TG_KERNEL_WENDLAND_C2, _abi.TG_POS_FP64)
        _check(rho.cpu().numpy(), cnt.cpu().numpy(), hs.cpu().numpy().view(np.uint64), o, 1e-12)


@pytest.mark.parametrize("dim", (2, 3))
@pytest.mark.parametrize("kernel", range(6))
def test_density_kernels(gpu_lib, dim, kernel):
    n, h, m = 700, 0.12, 0.5
    r = _cloud(n, dim, 0.0)
    scn = dict(dim=dim, tanks=[dict(n_fluid=n, n_wall=0, h=h, m=m, rho0=1000.0, cs0=1.0)],
               r=r, v=np.zeros_like(r), rho=np.full(n, 1000.0))
    with gpu_context(scn, physics.baseline_params(dim, kernel=kernel)) as ctx:
        for precision, tol in ((_abi.TG_POS_FP64, 1e-12), (_abi.TG_POS_FP32, 1e-5)):
            o = oracle.summation_density(r, h, m, kernel, precision)
            _check(*ctx.summation_density(precision), o, tol)
