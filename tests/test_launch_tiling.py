"""The z-operator products' row tiling is chosen per launch from the number of
column tiles; the solves must not depend on it.  Each grid's default (grids
that give one row tile, several, one m-tile per CTA; an even number of points,
which has dense operators only) against the fewest row tiles, set for every
launch through the autotuner's cache, bit for bit."""
import json

import numpy as np
import pytest

from oracle import turbid_oracle as O
from tests.test_gpu_parity import gpu_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 12, 5), (16, 12, 17), (32, 32, 65), (64, 48, 66), (96, 64, 98), (128, 128, 129),
                                   (256, 128, 65)])
def test_solves_do_not_depend_on_the_launch_tiling(cuda, tmp_path, shape):
    import torch
    nx, ny, nz = shape
    cfg = O.CaseConfig(nx=nx, ny=ny, nz=nz, bc_u=[1, 0, 0, 1, 0])
    gc = gpu_case(cfg)
    rng = np.random.default_rng(nz)
    rhs = torch.from_numpy(rng.standard_normal((nz, gc.M, 2))).to(cuda)
    path = tmp_path / "tiling.json"
    out = []
    for forced in (False, True):
        if forced:
            gc.autotune(str(path))
            (key, _), = json.loads(path.read_text()).items()
            path.write_text(json.dumps({key: [16, 6]}))
            gc.autotune(str(path))
        for which in (0, 2, 3):   # dense, split, split with the null mode
            y = torch.full_like(rhs, float("nan"))
            gc.helmholtz(which, 1, rhs.data_ptr(), y.data_ptr())
            out.append(y.cpu().numpy())
    gc.close()
    for a, b in zip(out[:3], out[3:]):
        assert np.array_equal(a, b)
