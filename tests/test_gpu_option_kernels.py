"""The kernels with the default options compiled in and the ones that read
them at run time, one option at a time on either side of the selection,
against the CPU oracle.

FP64 (-fmad=false) has to match bit for bit.  The mixed path's bound is that
of the other parity tests, 1e-5 in relative L1 density.
"""
import dataclasses

import numpy as np
import pytest

from flashx_b200 import amr as A
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


OPTIONS_3D = dict(OPTIONS, no_ctu={"use_3dFullCTU": False}, pressure_source={"hy_fPresInMomFlux": 0.5},
                  gravity={"useGravity": True, "gravity": (0.02, -0.03, -0.1)},
                  weno_gravity={"order": 5, "useGravity": True, "gravity": (0.02, -0.03, -0.1)})


@pytest.mark.parametrize("name", sorted(OPTIONS_3D))
def test_3d_option_matches_oracle(oracle, need_gpu, name):
    geom = Geometry(3, 8, 8, 8, 3, 2, 1,
                    bc=(BC_REFLECTING, BC_OUTFLOW, BC_PERIODIC, BC_PERIODIC, BC_REFLECTING, BC_REFLECTING))
    hp = dataclasses.replace(HydroParams(gamma=5.0 / 3.0), **OPTIONS_3D[name])
    _check(*_steps(oracle, geom, hp, S.noisy_gas(geom, hp)))


# extents where the sweeps' tiles and segments end unevenly: odd ones, the
# fewest cells a block can have, and one long axis at a time (several x
# segments, line segments and planes per CTA)
@pytest.mark.parametrize("order", [3, 5])
@pytest.mark.parametrize("shape", [((5, 6, 7), (2, 1, 3)), ((4, 4, 4), (1, 1, 1)), ((16, 4, 4), (11, 1, 1)),
                                   ((4, 16, 4), (1, 11, 1)), ((4, 4, 16), (1, 1, 11)), ((33, 9, 4), (1, 1, 1))])
def test_3d_sweep_extents_match_oracle(oracle, need_gpu, shape, order):
    (nx, ny, nz), (bx, by, bz) = shape
    for bc in ((BC_PERIODIC,) * 6, (BC_OUTFLOW,) * 2 + (BC_REFLECTING,) * 2 + (BC_PERIODIC,) * 2,
               (BC_REFLECTING,) * 2 + (BC_PERIODIC,) * 2 + (BC_OUTFLOW,) * 2):
        geom = Geometry(3, nx, ny, nz, bx, by, bz, bc=bc,
                        bbox=((0.0, float(nx * bx)), (0.0, float(ny * by)), (0.0, float(nz * bz))))
        hp = HydroParams(gamma=5.0 / 3.0, order=order)
        _check(*_steps(oracle, geom, hp, S.noisy_gas(geom, hp)))


# FP64 WENO5 with either set of kernels (the tuner would choose by time)
WENO_3D = {k: OPTIONS_3D[k] for k in ("weno", "weno_primitive", "weno_z", "weno_HLL", "weno_gravity")}
WENO_3D.update(weno_no_ctu={"order": 5, "use_3dFullCTU": False}, weno_flattening={"order": 5, "use_flattening": True},
               weno_pressure={"order": 5, "hy_fPresInMomFlux": 0.5})


@pytest.mark.parametrize("stages", ["0", "1"])
@pytest.mark.parametrize("name", sorted(WENO_3D))
def test_3d_weno_kernels_match_oracle(oracle, need_gpu, monkeypatch, name, stages):
    monkeypatch.setenv("FXB_WENO_STAGES", stages)
    geom = Geometry(3, 8, 8, 8, 3, 2, 1,
                    bc=(BC_REFLECTING, BC_OUTFLOW, BC_PERIODIC, BC_PERIODIC, BC_REFLECTING, BC_REFLECTING))
    hp = dataclasses.replace(HydroParams(gamma=5.0 / 3.0), **WENO_3D[name])
    unk = S.noisy_gas(geom, hp)
    dev = HydroDevice(geom, hp)
    dev.attach_unk(unk.copy())
    assert ("sweeps: per-stage kernels" if stages == "1" else "sweeps: one kernel per direction") in dev.tuning()
    dev.close()
    _check(*_steps(oracle, geom, hp, unk))


def _amr(oracle, geom, hp, maxlev=2, n=2, precisions=("fp64", "mixed")):
    """n steps of the level-set problem: (interiors per precision, oracle's, the last device's tuning text)."""
    mesh, unk = A.levelset_problem(geom, hp, maxlev)
    am = oracle.Amr(oracle.make_params(geom.as_dict(), hp), mesh.levels, mesh.bcoords)
    dt = 0.4 * am.compute_dt(unk)
    ref = unk.copy()
    for _ in range(n):
        am.hydro_step(ref, dt)
    g = geom.nguard
    out = {}
    for prec in precisions:
        dev = HydroDevice(geom, hp, prec, mesh=mesh)
        dev.attach_unk(unk.copy())
        for i in range(n):
            dev.Hydro(i * dt, dt, dt)
        o = unk.copy()
        dev.sync_to_host(o)
        log = dev.tuning()
        dev.close()
        out[prec] = o[:, g:-g, g:-g, g:-g][..., HYDRO_VARS]
    return out, ref[:, g:-g, g:-g, g:-g][..., HYDRO_VARS], log


# both forms of the step, and every branch of the sweep kernels' boundary fluxes
AMR_OPTIONS = {k: OPTIONS_3D[k] for k in ("default", "minmod", "vanLeer", "weno", "weno_HLL", "HLL", "no_ctu", "flattening",
                                          "pressure_source")}


@pytest.mark.parametrize("persistent", ["0", "1"])
@pytest.mark.parametrize("name", sorted(AMR_OPTIONS))
def test_amr_option_matches_oracle(oracle, need_gpu, monkeypatch, name, persistent):
    monkeypatch.setenv("FXB_AMR_PERSISTENT", persistent)
    geom = Geometry(3, 8, 8, 8, 2, 2, 2, bc=(BC_PERIODIC,) * 4 + (BC_REFLECTING,) * 2)
    hp = dataclasses.replace(HydroParams(), **AMR_OPTIONS[name])
    out, ref, log = _amr(oracle, geom, hp)
    assert ("step form: persistent" if persistent == "1" else "step form: batched launches") in log
    _check(out, ref)


# leaves that fill the sweeps' CTAs of 64, 96, 128 and 160 threads and ones
# that leave a remainder
@pytest.mark.parametrize("order,stages", [(3, "0"), (5, "0"), (5, "1")])
@pytest.mark.parametrize("n", [4, 6, 8, 10, 12, 16])
def test_amr_leaf_sizes_match_oracle(oracle, need_gpu, monkeypatch, n, order, stages):
    monkeypatch.setenv("FXB_AMR_PERSISTENT", "0")
    monkeypatch.setenv("FXB_WENO_STAGES", stages)
    geom = Geometry(3, n, n, n, 2, 1, 2, bc=(BC_PERIODIC,) * 2 + (BC_OUTFLOW,) * 2 + (BC_REFLECTING,) * 2)
    _check(*_amr(oracle, geom, HydroParams(order=order))[:2])


# more leaves than a batch takes: boundary fluxes stored in both passes; and
# the smaller CTAs of FP32 leaves, which only larger batches take
@pytest.mark.parametrize("opts", [{"slopeLimiter": "vanLeer"}, {"order": 5, "RiemannSolver": "HLL"},
                                  {"hy_fPresInMomFlux": 0.5}])
def test_amr_batches_of_sweeps_match_oracle(oracle, need_gpu, monkeypatch, opts):
    monkeypatch.setenv("FXB_AMR_PERSISTENT", "0")
    monkeypatch.setenv("FXB_AMR_MAX_BATCH", "23")
    geom = Geometry(3, 8, 8, 8, 2, 2, 2, bc=(BC_PERIODIC,) * 6)
    _check(*_amr(oracle, geom, dataclasses.replace(HydroParams(), **opts))[:2])


@pytest.mark.parametrize("order", [3, 5])
def test_amr_many_small_leaves_match_oracle(oracle, need_gpu, monkeypatch, order):
    monkeypatch.setenv("FXB_AMR_PERSISTENT", "0")
    geom = Geometry(3, 8, 8, 8, 3, 3, 3, bc=(BC_PERIODIC,) * 6)
    _check(*_amr(oracle, geom, HydroParams(order=order), maxlev=3, n=1)[:2])


# rows of whole 16-byte pairs, and (odd block sizes, odd slot counts) not;
# blocks of 935,088 and 1,068,672 bytes on both sides of the 1 MiB from which
# the copy engine moves them
@pytest.mark.parametrize("n", [8, 5, 21, 22])
def test_3d_interior_transfers_move_every_row(need_gpu, n):
    geom = Geometry(3, n, n + 1, n + 2, 3, 2, 2, bc=(BC_PERIODIC,) * 6)
    hp = HydroParams()
    unk = S.noisy_gas(geom, hp)
    dev = HydroDevice(geom, hp, "fp64")
    dev.attach_unk(unk.copy())
    other = unk.copy()
    other[..., DENS] *= 2.0
    dev.put_interior(other)
    got = np.full(geom.unk_shape, -7.0)
    dev.get_interior(got)
    g = geom.nguard
    inner = np.s_[:, g:-g, g:-g, g:-g]
    assert np.array_equal(got[inner][..., HYDRO_VARS], other[inner][..., HYDRO_VARS])
    got[inner] = -7.0
    assert np.all(got == -7.0), "guard cells keep their values"
    dev.close()
