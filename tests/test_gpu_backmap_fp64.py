"""The FP64 backmap at the edges of its tiles (128 samples x 64 outputs x 16
deep), both sample types, rows that allow 16-byte copies and rows that do not
(GPU).  Tolerance: d + 2 roundings of half an ulp each, (d + 2) 2^-53 of
sum_k |T_ik y_k| + |shift_i|."""
import numpy as np
import pytest

from naja_b200 import backmap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(1, 1, 1), (127, 63, 15), (128, 64, 16), (129, 66, 20), (257, 65, 17), (300, 130, 48),
                                   (640, 200, 100)])
def test_tile_edges(cuda, shape, dtype):
    N, n, d = shape
    rng = np.random.default_rng(N)
    T, shift = rng.standard_normal((n, d)), rng.standard_normal(n)
    Y = (rng.standard_normal((N, d)) * 10 ** rng.uniform(-2, 2, (1, d))).astype(dtype)
    V = backmap(T, shift, Y, mode="fp64", out_dtype=np.float64)
    y = Y.astype(np.longdouble)
    ref = y @ T.astype(np.longdouble).T + shift
    scale = np.abs(y) @ np.abs(T).T + np.abs(shift)
    assert np.max(np.abs(V - ref) / scale) <= (d + 2) * 2.0 ** -53
    assert np.array_equal(backmap(T, shift, Y, mode="fp64", out_dtype=np.float32), V.astype(np.float32))
