"""Performance cases of turbid_b200: the work a user of the library has it do,
through the public Python classes and the C ABI they wrap.

Kinds
  run        a restart job: the restart state is uploaded from pinned host
             memory, a number of RK3 steps runs (tg_run_steps), the state is
             downloaded into pinned host memory;
  plugin     the same job through the per-stage plugin methods, as the main
             program's FlatChannelSolver::Execute loop calls them (one call per
             phase method and stage, the features read after every step);
  ensemble   independent cases on uneven grids stepped together, each from and
             to its own pinned host buffers;
  transform  the field container's plane transforms on device buffers, forward
             then backward (whole fields, or the planes of a z-slab);
  helmholtz  the z-solves of u, w and the pressure on device buffers.

Grids run from 32x32x65 to 512x256x257, the sizes of the benchmark's
workloads: powers of two, the other lengths with small prime factors that
spectral cases use, and now and then any length.  Jobs in mixed precision
carry FP32 accuracy in every field (FP32 transforms and products), so the job
keeps its downloaded fields as a single-precision snapshot; FP64 jobs keep
the FP64 fields.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import turbid_b200 as tb
from turbid_b200 import _lib, synthetic
from turbid_b200.solver import run_ensemble

# the oscillatory boundary layer of the benchmark (Stokes-layer units)
_FLOW = dict(lx=4 * math.pi, ly=2 * math.pi, dt=2 * math.pi / 2000, reynolds=800.0, froude=1.0,
             averaged_concentration=1e-3, specific_gravity=2.65, affected_by_scalar=1, bc_u=[1, 0, 0, 1, 0],
             bc_v=[1, 0, 0, 1, 0], bc_w=[1, 0, 1, 0, 0], bc_p=[0, 1, 0, 1, 0], force_type=2,
             force_direction=[0, 1], force_amplitude=[0, 1], schmidt=0.5, settling=5e-4, erosion_rate=1e-4,
             critical_shear=2e-4, scalar_bc=1)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed() -> list:
    return [
        # a laminar validation job: the smallest grid, carrier phase only, FP64
        _run("laminar_32x32x65_fp64", 32, 32, 65, "fp64", 1, 20, reynolds=180.0),
        # an interactive job on a small sediment case, stepped through the plugin methods
        dict(name="plugin_64x64x65_mixed", kind="plugin", nx=64, ny=64, nz=65, precision="mixed", nphase=2, steps=4,
             reynolds=800.0, scalar_bc=1),
        # the parity-mode sediment case
        _run("sediment_128x128x129_fp64", 128, 128, 129, "fp64", 2, 10),
        # a parity-mode case on a grid with factors of three and five, no-flux bed
        _run("sediment_120x96x81_fp64", 120, 96, 81, "fp64", 2, 6, scalar_bc=0),
        # the benchmark's headline grid, mixed precision
        _run("sediment_256x256x257_mixed", 256, 256, 257, "mixed", 2, 20),
        # the largest single case: a longer domain
        _run("sediment_512x256x257_mixed", 512, 256, 257, "mixed", 2, 10, reynolds=1000.0),
        # a parameter study: uneven cases stepped together
        dict(name="ensemble_64_to_192_mixed", kind="ensemble", grids="64x65 80x81 96x97 120x121 144x145 192x193",
             precision="mixed", steps=5),
        # whole velocity fields in double precision, power-of-two planes
        dict(name="transform_256x256_fp64", kind="transform", nx=256, ny=256, planes=771, precision="fp64"),
        # whole velocity fields in single precision, planes with a factor of three
        dict(name="transform_192x192_fp32", kind="transform", nx=192, ny=192, planes=579, precision="fp32"),
        # one rank's z-slab of a distributed case on an uneven grid
        dict(name="slab_250x90_fp64", kind="transform", nx=250, ny=90, planes=21, precision="fp64"),
        # the wall planes of a small case: the smallest call
        dict(name="planes_64x64_fp32", kind="transform", nx=64, ny=64, planes=2, precision="fp32"),
        # the z-solves of one stage in double precision
        dict(name="helmholtz_128x128x129_fp64", kind="helmholtz", nx=128, ny=128, nz=129, precision="fp64"),
    ]


def _run(name, nx, ny, nz, precision, nphase, steps, reynolds=800.0, scalar_bc=1) -> dict:
    return dict(name=name, kind="run", nx=nx, ny=ny, nz=nz, precision=precision, nphase=nphase, steps=steps,
                reynolds=reynolds, scalar_bc=scalar_bc)


def _smooth(n: int) -> bool:
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


def _length(rng, lo: int, hi: int) -> int:
    """A transform length, spread over the logarithm: mostly even with small
    prime factors, a quarter powers of two, some of any factors and parity."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.random()
    if kind < 0.25:
        return max(lo, min(hi, 1 << int(round(math.log2(n)))))
    if kind < 0.85:
        return min((m for m in range(lo, hi + 1, 2) if _smooth(m)), key=lambda m: abs(m - n))
    return n if kind < 0.93 else min(hi - hi % 2, n + n % 2)


def _height(rng, lo: int, hi: int) -> int:
    """Chebyshev points: an odd number (an even count of intervals), at times even."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.12:
        return n - n % 2
    kind = rng.random()
    if kind < 0.4:
        return (1 << int(round(math.log2(n)))) + 1
    if kind < 0.8:
        return min((m for m in range(lo, hi + 1, 2) if _smooth(m - 1)), key=lambda m: abs(m - n))
    return n | 1


def draw(rng) -> dict:
    kind = rng.choice(["run", "run", "run", "plugin", "ensemble", "transform", "transform", "transform", "helmholtz"])
    if kind == "transform":
        nx, ny = _length(rng, 32, 512), _length(rng, 32, 512)
        most = max(1, min(771, 50_000_000 // (nx * ny)))
        if not (_smooth(nx) and _smooth(ny)):
            most = max(1, most // 8)
        planes = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
        return dict(kind=kind, nx=nx, ny=ny, planes=planes, precision=rng.choice(["fp64", "fp32"]))
    if kind == "helmholtz":
        nx, ny = _length(rng, 32, 256), _length(rng, 32, 256)
        return dict(kind=kind, nx=nx, ny=ny, nz=_height(rng, 33, 257), precision=rng.choice(["fp64", "mixed"]))
    if kind == "ensemble":
        sizes = [n for n in range(64, 161, 2) if _smooth(n)]
        grids = " ".join("%dx%d" % (n, n + 1) for n in (rng.choice(sizes) for _ in range(rng.randint(2, 4))))
        return dict(kind=kind, grids=grids, precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(1, 4))
    nx, ny = _length(rng, 32, 320), _length(rng, 32, 256)
    nz = _height(rng, 33, 257)
    budget = 40_000_000 if _smooth(nx) and _smooth(ny) else 8_000_000   # points times steps
    steps = max(1, min(rng.randint(1, 12), budget // (nx * ny * nz)))
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=rng.choice(["fp64", "mixed"]), nphase=rng.choice([1, 2, 2]),
                steps=steps, reynolds=round(rng.uniform(180.0, 1000.0), 1), scalar_bc=rng.choice([0, 1]))


# ---------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------
def _pinned(a: np.ndarray) -> np.ndarray:
    """A pinned host copy of a complex array (as numpy, sharing the pinned memory)."""
    t = torch.empty(2 * a.size, dtype=torch.float64, pin_memory=True)
    out = t.numpy().view(np.complex128).reshape(a.shape)
    out[...] = a
    return out


def _job(params: dict, seed: int) -> dict:
    """One case with its restart state in pinned host memory."""
    case = tb.ChannelCase(**params)
    stream = torch.cuda.Stream()   # steps replay as graphs off the legacy default stream
    case.set_stream(stream.cuda_stream)
    init = [_pinned(a) for a in synthetic.initial_state(seed=seed, **params)]
    if params["nphase"] == 1:
        init = init[:2]
    single = params["precision"] == "mixed"
    host = [torch.empty(2 * a.size, dtype=torch.float64, pin_memory=True) for a in init]
    snap = [torch.empty(2 * a.size, dtype=torch.float32) for a in init] if single else host
    return dict(case=case, stream=stream, init=init, host=host, snap=snap, single=single, shapes=[a.shape for a in init],
                features=np.zeros(_lib.TG_NFEATURE), dt=params["dt"])


def _params(case: dict) -> dict:
    return dict(_FLOW, **{k: case[k] for k in ("nx", "ny", "nz", "precision", "nphase", "reynolds", "scalar_bc")})


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("run", "plugin"):
        return dict(kind=kind, steps=case["steps"], nphase=case["nphase"], jobs=[_job(_params(case), seed)])
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        jobs = []
        for i, g in enumerate(case["grids"].split()):
            n, nz = (int(v) for v in g.split("x"))
            p = dict(_FLOW, nx=n, ny=n, nz=nz, nphase=2, precision=case["precision"],
                     reynolds=float(rng.uniform(400.0, 1000.0)), settling=float(10 ** rng.uniform(-4.0, -3.0)))
            jobs.append(_job(p, seed + 1000 * i))
        return dict(kind=kind, steps=case["steps"], jobs=jobs)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "transform":
        fp32 = case["precision"] == "fp32"
        # the handle of the case whose planes these are: three fields, or a slab of one
        nz = max(33, min(257, case["planes"] // 3))
        h = tb.ChannelCase(**dict(_FLOW, nx=case["nx"], ny=case["ny"], nz=nz, nphase=1,
                                  precision="mixed" if fp32 else "fp64"))
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        phys = _phys(case, gen)
        spec = torch.empty((case["planes"], h.M), dtype=torch.complex128, device="cuda")
        return dict(kind=kind, h=h, phys=phys, spec=spec, back=torch.empty_like(phys), planes=case["planes"], fp32=fp32)
    h = tb.ChannelCase(**dict(_FLOW, nx=case["nx"], ny=case["ny"], nz=case["nz"], nphase=1, precision=case["precision"]))
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    rhs = _rhs(case, gen)
    return dict(kind=kind, h=h, rhs=rhs, out=torch.empty_like(rhs))


def _phys(case: dict, gen) -> torch.Tensor:
    """Velocity-like planes: a mean of order one plus fluctuations."""
    dtype = torch.float32 if case["precision"] == "fp32" else torch.float64
    shape = (case["planes"], case["ny"], case["nx"])
    mean = torch.rand((shape[0], 1, 1), generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    return (mean + 0.1 * torch.randn(shape, generator=gen, device="cuda", dtype=dtype)).to(dtype)


def _rhs(case: dict, gen) -> torch.Tensor:
    """Right-hand sides of u, w and the pressure: decaying spectra."""
    m = (case["ny"] // 3 * 2) * (case["nx"] // 3 * 2 // 2 + 1)
    r = torch.randn((3, case["nz"], m, 2), generator=gen, device="cuda", dtype=torch.float64)
    decay = 1.0 / (1.0 + torch.arange(m, device="cuda", dtype=torch.float64) / 64.0)
    return torch.view_as_complex(r * decay[None, None, :, None])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _upload(j: dict):
    a = j["init"]
    j["case"].upload_state(a[0], a[1], a[2] if len(a) > 2 else None)


def _download(j: dict) -> list:
    c = j["case"]
    ptr = [t.data_ptr() for t in j["host"]] + [None]
    pd = _lib._pd
    cast = _lib.ctypes.cast
    _lib.check(c.lib.tg_download_state(c.h, *[None if p is None else cast(p, pd) for p in ptr[:3]]))
    if j["single"]:
        for dst, src in zip(j["snap"], j["host"]):
            dst.copy_(src)
    return [torch.view_as_complex(t.view(*s, 2)) for t, s in zip(j["snap"], j["shapes"])]


def run(state):
    kind = state["kind"]
    if kind == "transform":
        h, n, fp32 = state["h"], state["planes"], state["fp32"]
        h.dft_forward_planes(state["phys"].data_ptr(), state["spec"].data_ptr(), n, fp32=fp32)
        h.dft_backward_planes(state["spec"].data_ptr(), state["back"].data_ptr(), n, fp32=fp32)
        # in single precision the spectral planes hold the FP32 values of the round trip
        return [state["back"]] if fp32 else [state["back"], state["spec"]]
    if kind == "helmholtz":
        h, rhs, out = state["h"], state["rhs"], state["out"]
        for i, which in enumerate((0, 2, 3)):
            h.helmholtz(which, 1, rhs[i].data_ptr(), out[i].data_ptr())
        return [out[0], out[1], out[2]]
    jobs, steps = state["jobs"], state["steps"]
    for j in jobs:
        _upload(j)
    if kind == "run":
        jobs[0]["case"].run_steps(steps)
    elif kind == "ensemble":
        run_ensemble([j["case"] for j in jobs], steps)
    else:   # the Execute loop over the plugin methods
        c, dt = jobs[0]["case"], jobs[0]["dt"]
        for n in range(steps):
            c.set_time(n + 1, (n + 1) * dt, dt, n % 2 == 1)
            for stage in range(3):
                c.carrier_predict(stage)
                c.carrier_correct(stage)
                if state["nphase"] > 1:
                    c.scalar_predict(stage)
                    c.scalar_correct(stage)
            c.features()
    return [_download(j) for j in jobs]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _modes(nx: int, ny: int) -> int:
    return (ny // 3 * 2) * (nx // 3 * 2 // 2 + 1)


def _step_work(nx: int, ny: int, nz: int, nphase: int) -> tuple:
    """One RK3 step: per stage the spectral state (velocity, pressure, scalar
    and the registers) read and written once; the fewest plane transforms of
    either nonlinear form (3 velocities back, 3 advection terms forward; the
    scalar's field back, its advection and filtered field forward) and the
    reference's two dense products of every Helmholtz solve."""
    m, pts = _modes(nx, ny), nx * ny * nz
    fields = 4 + 3 + (2 if nphase > 1 else 0)
    transforms = 6 + (3 if nphase > 1 else 0)
    solves = 4 + (1 if nphase > 1 else 0)
    by = fields * 2 * 16.0 * nz * m
    fl = transforms * 2.5 * pts * math.log2(nx * ny) + solves * 2 * 4.0 * nz * nz * m
    return 3 * by, 3 * fl


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "transform":
        m, pts = _modes(case["nx"], case["ny"]), case["nx"] * case["ny"]
        real = 4 if case["precision"] == "fp32" else 8
        return {"bytes": 2.0 * case["planes"] * (pts * real + 16 * m),
                "flops": 2 * case["planes"] * 2.5 * pts * math.log2(pts)}
    if kind == "helmholtz":
        m = _modes(case["nx"], case["ny"])
        return {"bytes": 3 * 2 * 16.0 * case["nz"] * m, "flops": 3 * 2 * 4.0 * case["nz"] ** 2 * m}
    if kind == "ensemble":
        grids = [tuple(int(v) for v in g.split("x")) for g in case["grids"].split()]
        grids = [(n, n, nz, 2) for n, nz in grids]
    else:
        grids = [(case["nx"], case["ny"], case["nz"], case["nphase"])]
    by = fl = 0.0
    for nx, ny, nz, nphase in grids:
        b, f = _step_work(nx, ny, nz, nphase)
        state = (4 + nphase - 1) * 16.0 * nz * _modes(nx, ny)
        by += case["steps"] * b + 2 * state
        fl += case["steps"] * f
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# the values in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def exact(case: dict, seed: int):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "transform":
        nx, ny = case["nx"], case["ny"]
        nyc, nxh = ny // 3 * 2, nx // 3 * 2 // 2 + 1
        low, high = nyc // 2, nyc - nyc // 2
        full = torch.fft.rfft2(_phys(case, gen).double(), norm="forward")[:, :, :nxh]
        kept = torch.cat([full[:, :low], full[:, ny - high:]], dim=1)          # (planes, nyc, nxh)
        pad = torch.zeros((case["planes"], ny, nx // 2 + 1), dtype=torch.complex128, device="cuda")
        pad[:, :low, :nxh], pad[:, ny - high:, :nxh] = kept[:, :low], kept[:, low:]
        cols = torch.fft.ifft(pad, dim=1, norm="forward")
        cols[:, :, 0] = cols[:, :, 0].real.to(torch.complex128)
        back = torch.fft.irfft(cols, n=nx, dim=2, norm="forward")
        spec = kept.transpose(1, 2).reshape(case["planes"], -1)
        return [back] if case["precision"] == "fp32" else [back, spec]
    if kind == "helmholtz":
        return _exact_helmholtz(case, gen)
    return None


def _exact_helmholtz(case: dict, gen):
    """Direct solves of the collocation systems of u and w, mode by mode:
    (D2 + kx2 + ky2 + sigma) x = rhs inside, the boundary conditions' rows at
    the walls (u: value below, slope above; w: values)."""
    nx, ny, n = case["nx"], case["ny"], case["nz"]
    m = _modes(nx, ny)
    if m * float(n) ** 3 > 4e10:
        return None
    z = np.cos((n - 1 - np.arange(n)) * np.pi / (n - 1))
    c = np.ones(n)
    c[0] = c[-1] = 2.0
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    with np.errstate(divide="ignore", invalid="ignore"):
        d1 = np.where(i == j, 0.0, c[i] / c[j] * (-1.0) ** (i + j) / (z[i] - z[j]))
    np.fill_diagonal(d1, -d1.sum(axis=1))
    d2 = d1 @ d1
    np.fill_diagonal(d2, 0.0)
    np.fill_diagonal(d2, -d2.sum(axis=1))
    nyc, nxh = ny // 3 * 2, nx // 3 * 2 // 2 + 1
    kx = 2 * np.pi / _FLOW["lx"] * np.arange(nxh)
    iy = np.arange(nyc)
    ky = 2 * np.pi / _FLOW["ly"] * np.where(iy <= nyc // 2, iy, iy - nyc)
    shift = -(kx[:, None] ** 2 + ky[None, :] ** 2).reshape(-1) - _FLOW["reynolds"] / _FLOW["dt"] / (5.0 / 24.0)
    D1, D2, s = (torch.from_numpy(a).cuda() for a in (d1, d2, shift))
    rhs = _rhs(case, gen)
    out = []
    for f, top in ((0, D1[n - 1]), (1, torch.eye(n, dtype=torch.float64, device="cuda")[n - 1])):
        x = torch.empty_like(rhs[f])
        for m0 in range(0, m, 512):
            m1 = min(m, m0 + 512)
            A = D2[None] + s[m0:m1, None, None] * torch.eye(n, dtype=torch.float64, device="cuda")
            A[:, 0] = 0.0
            A[:, 0, 0] = 1.0
            A[:, n - 1] = top
            b = torch.view_as_real(rhs[f, :, m0:m1].transpose(0, 1).contiguous())
            sol = torch.linalg.solve(A, b)
            x[:, m0:m1] = torch.view_as_complex(sol.contiguous()).transpose(0, 1)
        out.append(x)
    return [out[0], out[1], None]
