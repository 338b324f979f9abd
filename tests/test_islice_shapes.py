"""The int8-slice product at the edges of its shapes: the K steps in use (32
interior rows each, four to a half tile), the operator's 96-row chunks (a last
chunk of few rows, of one 16-row step, of more than 64 rows) and the smallest
grids, bit for bit against the numpy model of its arithmetic."""
import ctypes

import numpy as np
import pytest

import turbid_b200 as tb
from tests.test_islice import _case, _data, islice_model
from turbid_b200 import _lib

pytestmark = pytest.mark.gpu


# interior rows nz - 2: 3, 32, 33, 96, 128, 129, 160, 161, 192, 193, 224, 225, 256;
# output rows nz: chunks of 96 with 5, 34, 35, 2, 34, 35, 66, 67, 2, 3, 34, 35, 66 in the last
@pytest.mark.parametrize("nz", [5, 34, 35, 98, 130, 131, 162, 163, 194, 195, 226, 227, 258])
def test_product_matches_model_bitwise(cuda, nz):
    import torch
    gc = _case(24, 18, nz)
    gc.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(nz)
    X = _data(rng, nz, 2 * gc.M)[None]
    A = np.ascontiguousarray(rng.standard_normal((nz, nz)) * 10.0 ** rng.uniform(-3, 3, nz)[:, None])
    xd = torch.from_numpy(X.copy()).to(cuda)
    yd = torch.full_like(xd, float("nan"))
    _lib.check(_lib.load().tg_multiply_islice(gc.h, A.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                              ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(yd.data_ptr()), 1))
    got = yd.cpu().numpy()[0]
    assert np.array_equal(got, islice_model(A, X[0])), nz
    gc.close()
