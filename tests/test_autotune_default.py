"""tg_autotune and the row tiling chosen per launch: the per-launch choice is a
candidate of the tuner, so a tuned context is no slower than an untuned one at
one component or at three, and a cache can say "per launch" (a preference of 0,
or the m-tiles that choice takes at three components)."""
import json

import numpy as np
import pytest

import turbid_b200 as tb
from oracle import turbid_oracle as O
from tests.test_gpu_parity import gpu_case

pytestmark = pytest.mark.gpu


def _solves(cuda, gc, cfg):
    import torch
    rhs = torch.from_numpy(np.random.default_rng(3).standard_normal((cfg.nz, gc.M, 2))).to(cuda)
    out = []
    for which in (0, 2, 3):
        y = torch.full_like(rhs, float("nan"))
        gc.helmholtz(which, 1, rhs.data_ptr(), y.data_ptr())
        out.append(y.cpu().numpy())
    return out


@pytest.mark.parametrize("nz", [33, 34])   # folded and dense operators; dense only
def test_zero_preferences_are_the_untuned_default(cuda, tmp_path, nz):
    cfg = O.CaseConfig(nx=32, ny=24, nz=nz, bc_u=[1, 0, 0, 1, 0])
    gc = gpu_case(cfg)
    ref = _solves(cuda, gc, cfg)
    path = tmp_path / "tiling.json"
    gc.autotune(str(path))
    (key, entry), = json.loads(path.read_text()).items()
    reported = []
    for prefs in ([0, 0], [0, 6], [16, 0], [-1, 0], [0, 7], entry):
        path.write_text(json.dumps({key: prefs}))
        if min(prefs) < 0 or prefs[1] > 6:
            with pytest.raises(tb.TgError, match="out of range"):
                gc.autotune(str(path))
            continue
        reported.append(gc.autotune(str(path)))
        assert json.loads(path.read_text()) == {key: prefs}   # applied, not timed again
        for a, b in zip(ref, _solves(cuda, gc, cfg)):
            assert np.array_equal(a, b)
    need = (nz + 7) // 8
    assert (reported[2]["mt_dense"], reported[2]["tiles_dense"]) == (need, 1)   # 16: one row tile
    # "per launch" reports the tiling of a three-component launch, and that
    # tiling's m-tiles stand for it
    assert all(v >= 1 for v in reported[0].values())
    path.write_text(json.dumps({key: [reported[0]["mt_dense"], reported[0]["mt_folded"]]}))
    assert gc.autotune(str(path)) == reported[0]
    gc.close()


def test_entries_of_the_former_tuner_are_timed_again(cuda, tmp_path):
    """Entries without the tuner's version in the key came from a tuner that
    pinned the best fixed tiling; they stay in the file."""
    cfg = O.CaseConfig(nx=32, ny=24, nz=33)
    gc = gpu_case(cfg)
    path = tmp_path / "tiling.json"
    gc.autotune(str(path))
    (key, entry), = json.loads(path.read_text()).items()
    assert key.startswith("32x24x33:fp64:sm") and key.endswith(":2")
    path.write_text(json.dumps({key[:-2]: [16, 6]}))
    gc.autotune(str(path))
    cache = json.loads(path.read_text())
    assert cache[key[:-2]] == [16, 6] and set(cache) == {key, key[:-2]}
    gc.close()


# grids on which the best fixed tiling at three components costs a
# single-component launch 40-80 %
@pytest.mark.parametrize("shape", [(64, 64, 129), (128, 128, 257)])
def test_tuned_solves_are_not_slower(cuda, shape):
    """Device time of single-component solves (dense, split) before and after
    the tuner: a fixed tiling is taken only where it is faster than the
    per-launch one, so 15 % covers the scatter of the timings."""
    import torch
    nx, ny, nz = shape
    gc = gpu_case(O.CaseConfig(nx=nx, ny=ny, nz=nz, bc_u=[1, 0, 0, 1, 0]))
    stream = torch.cuda.Stream()
    gc.set_stream(stream.cuda_stream)
    rhs = torch.from_numpy(np.random.default_rng(5).standard_normal((nz, gc.M, 2))).to(cuda)
    out = torch.empty_like(rhs)
    torch.cuda.synchronize()

    def least(which):
        best = float("inf")
        with torch.cuda.stream(stream):
            for _ in range(12):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(20):
                    gc.helmholtz(which, 1, rhs.data_ptr(), out.data_ptr())
                b.record()
                b.synchronize()
                best = min(best, a.elapsed_time(b))
        return best

    before = [least(w) for w in (0, 2)]
    gc.autotune(None)
    after = [least(w) for w in (0, 2)]
    gc.close()
    assert all(t <= 1.15 * s for s, t in zip(before, after)), (before, after)
