"""Whole steps on the grids whose transform passes no other step test reaches:
FP64 against the oracle at 256 points (the advection sums on 16-point last
butterflies) and with odd Ny beside a power of two or an even smooth Nx (a row
pair whose second row does not exist); mixed precision against FP64 at lengths
of three and four passes, in x and in y, with the same odd Ny.

Two steps are both nonlinear forms, the scalar's among them.  Tolerances as for
every step test: FP64 1e-10 (oracle), mixed 1e-5 (FP64), relative L2 per field.
"""
import pytest

from oracle import turbid_oracle as O
from tests.test_gpu_parity import gpu_case, rel, sediment_cfg

pytestmark = pytest.mark.gpu


def _fields(gc, state):
    gc.upload_state(*state)
    gc.run_steps(2)
    u, p, c = gc.download_state()
    gc.close()
    return {"u": u[0], "v": u[1], "w": u[2], "p": p, "c": c}


@pytest.mark.parametrize("shape", [(256, 18, 9), (32, 27, 9), (64, 21, 9), (18, 15, 9)])
def test_fp64_steps_match_oracle(cuda, shape):
    nx, ny, nz = shape
    cfg = sediment_cfg(nx=nx, ny=ny, nz=nz)
    state = O.make_initial_state(cfg, seed=31, noise=0.05)
    sol = O.OracleSolver(cfg, *state)
    got = _fields(gpu_case(cfg), state)
    for _ in range(2):
        sol.run_step()
    ref = {"u": sol.uvw[0], "v": sol.uvw[1], "w": sol.uvw[2], "p": sol.p, "c": sol.phi}
    errs = {k: rel(got[k], ref[k]) for k in ref}
    assert all(e < 1e-10 for e in errs.values()), errs


@pytest.mark.parametrize("shape", [(192, 24, 17), (250, 18, 17), (500, 18, 17), (32, 27, 17), (18, 15, 17),
                                   (18, 250, 17), (32, 500, 17)])
def test_mixed_steps_match_fp64(cuda, shape):
    nx, ny, nz = shape
    cfg = sediment_cfg(nx=nx, ny=ny, nz=nz)
    state = O.make_initial_state(cfg, seed=32, noise=0.05)
    ref, got = (_fields(gpu_case(cfg, precision), state) for precision in ("fp64", "mixed"))
    errs = {k: rel(got[k], ref[k]) for k in ref}
    assert all(e < 1e-5 for e in errs.values()), errs
