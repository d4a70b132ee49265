"""The kernels with the default options compiled in and the ones that read
them at run time, one option at a time on either side of the selection,
against the CPU oracle.

FP64 (-fmad=false) has to match bit for bit.  The mixed path's bound is that
of the other parity tests, 1e-5 in relative L1 density.
"""
import dataclasses

import numpy as np
import pytest

from flashx_b200 import simulations as S
from flashx_b200.hydro import HydroDevice
from flashx_b200.params import (BC_OUTFLOW, BC_PERIODIC, BC_REFLECTING, DENS, EINT, ENER, GAMC, GAME,
                                Geometry, HydroParams, PRES, TEMP, VELX, VELY, VELZ)

pytestmark = pytest.mark.gpu

HYDRO_VARS = [DENS, EINT, ENER, GAMC, GAME, PRES, TEMP, VELX, VELY, VELZ]
L1_TOL_MIXED = 1e-5

OPTIONS = {
    "default": {},
    "minmod": {"slopeLimiter": "minmod"},
    "vanLeer": {"slopeLimiter": "vanLeer"},
    "hybrid": {"slopeLimiter": "hybrid"},
    "limited": {"slopeLimiter": "limited"},
    "primitive": {"charLimiting": False},
    "HLL": {"RiemannSolver": "HLL"},
    "LLF": {"RiemannSolver": "LLF"},
    "no_aux_eint": {"use_auxEintEqn": False},
    "flattening": {"use_flattening": True},
    "weno": {"order": 5},
    "weno_minmod": {"order": 5, "slopeLimiter": "minmod"},     # the limiter is not used: default kernels
    "weno_primitive": {"order": 5, "charLimiting": False},
    "weno_z": {"order": 5, "wenoMethod": "WENOZ"},
    "weno_HLL": {"order": 5, "RiemannSolver": "HLL"},
}


def _steps(oracle, geom, hp, unk, n=2):
    """n steps on the device in both precisions and with the oracle."""
    p = oracle.make_params(geom.as_dict(), hp)
    dt = 0.4 * oracle.compute_dt(p, unk)
    ref = unk.copy()
    for _ in range(n):
        oracle.hydro_step(p, ref, dt, dt)
    out = {}
    for prec in ("fp64", "mixed"):
        dev = HydroDevice(geom, hp, prec)
        dev.attach_unk(unk.copy())
        for i in range(n):
            dev.Hydro(i * dt, dt, dt)
        o = np.zeros(geom.unk_shape)
        dev.sync_to_host(o)
        dev.close()
        out[prec] = S.gather_global(geom, o)[..., HYDRO_VARS]
    return out, S.gather_global(geom, ref)[..., HYDRO_VARS]


def _check(out, ref):
    assert np.array_equal(out["fp64"], ref)
    d, r = out["mixed"][..., 0], ref[..., 0]
    assert np.mean(np.abs(d - r)) / np.mean(np.abs(r)) <= L1_TOL_MIXED


@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_2d_option_matches_oracle(oracle, need_gpu, name):
    # 3 x 2 tiles: every tile at an edge, a different boundary on each axis
    geom = Geometry(2, 16, 16, 1, 3, 2, 1, bc=(BC_REFLECTING, BC_OUTFLOW, BC_PERIODIC, BC_PERIODIC) + (BC_OUTFLOW,) * 2)
    hp = dataclasses.replace(HydroParams(gamma=5.0 / 3.0), **OPTIONS[name])
    _check(*_steps(oracle, geom, hp, S.noisy_gas(geom, hp)))
