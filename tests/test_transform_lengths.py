"""Plane transforms of the even lengths with prime factors up to 7 (compiled
radices, turbid_b200/csrc/fft_mr_impl.cuh) against the oracle, and the
nonlinear terms formed inside their x passes against the oracle's RK3 step.

Tolerances as for the other transforms (tests/test_gpu_parity.py): FP64 1e-13,
FP32 3e-6, FP64 steps 1e-10 relative L2.
"""
import numpy as np
import pytest

import turbid_b200 as tb
from oracle import turbid_oracle as O
from tests.test_gpu_parity import gpu_case, rel, sediment_cfg

pytestmark = pytest.mark.gpu


def smooth(n):
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


# every length up to the largest, x and y paired from the two ends; the first
# ones below (16, 14) and above (540) the compiled range, and the neighbours of
# powers of two (a power of two in one direction only)
LENGTHS = [n for n in range(18, 513, 2) if smooth(n) and n & (n - 1)]
PAIRS = list(zip(LENGTHS, reversed(LENGTHS))) + [(14, 18), (540, 18), (18, 540), (64, 96), (96, 64), (18, 7), (9, 18)]


@pytest.mark.parametrize("fp32", [False, True])
def test_lengths_match_oracle(cuda, fp32):
    import torch
    for i, (nx, ny) in enumerate(PAIRS):
        nz = 3
        cfg = O.CaseConfig(nx=nx, ny=ny, nz=nz)
        g = O.Grid(cfg)
        gc = gpu_case(cfg, "mixed" if fp32 else "fp64")
        x = np.random.default_rng(i).standard_normal((1, nz, ny, nx))
        if fp32:
            x = x.astype(np.float32).astype(np.float64)
        ref = O.dft_forward(g, x)
        xd = torch.from_numpy(x).to(cuda, torch.float32 if fp32 else torch.float64)
        sd = torch.zeros((1, nz, g.M), dtype=torch.complex128, device=cuda)
        gc.dft_forward(xd.data_ptr(), sd.data_ptr(), 1, fp32=fp32)
        tol = 3e-6 if fp32 else 1e-13
        assert rel(tb.from_slab(sd.cpu().numpy(), g.nxh, g.nyc), ref) < tol, (nx, ny)
        # a spectral field whose kx = 0 plane is not Hermitian: c2r drops that part
        s = np.random.default_rng(1000 + i).standard_normal((2, 1, g.nxh, g.nyc, nz))
        spec = s[0] + 1j * s[1]
        sd.copy_(torch.from_numpy(tb.to_slab(spec)).reshape(sd.shape))
        xb = torch.zeros_like(xd)
        gc.dft_backward(sd.data_ptr(), xb.data_ptr(), 1, fp32=fp32)
        assert rel(xb.cpu().numpy().astype(np.float64), O.dft_backward(g, spec)) < tol, (nx, ny)
        gc.close()


@pytest.mark.parametrize("shape", [(18, 20, 17), (36, 18, 9), (32, 18, 17), (18, 32, 17), (18, 14, 17), (14, 18, 17),
                                   (250, 18, 9), (18, 196, 9)])
def test_steps_match_oracle(cuda, shape):
    """Both nonlinear forms (two steps), the scalar's among them."""
    nx, ny, nz = shape
    cfg = sediment_cfg(nx=nx, ny=ny, nz=nz)
    uvw, p, phi = O.make_initial_state(cfg, seed=21, noise=0.05)
    sol = O.OracleSolver(cfg, uvw, p, phi)
    gc = gpu_case(cfg)
    gc.upload_state(uvw, p, phi)
    for _ in range(2):
        gc.run_steps(1)
        sol.run_step()
    u, pp, c = gc.download_state()
    errs = {"u": rel(u, sol.uvw), "p": rel(pp, sol.p), "c": rel(c, sol.phi)}
    gc.close()
    assert all(v < 1e-10 for v in errs.values()), errs
