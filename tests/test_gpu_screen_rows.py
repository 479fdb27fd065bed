"""The screened dense kernel at its largest row counts and its final slack (GPU),
bit for bit: samples against the CPU oracle, slack against the kernel that
divides every row."""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import Polytope

pytestmark = pytest.mark.gpu


def _polytope(m, d, seed):
    rng = np.random.default_rng(seed)
    half = rng.standard_normal(((m + 1) // 2, d))
    return np.concatenate([half, -half])[:m], 10.0 ** rng.uniform(0.0, 2.0, m)


def _run(P, **kw):
    dt = np.float64 if kw["precision"] == "fp64" else np.float32
    sf = np.empty((3, P.m), dt)
    S = P.run(np.zeros(P.d), 15, 3, 3, seed=5, pair_prob=0.4, resync_interval=11, out_dtype="f64", sparse="dense",
              slack_final=sf, **kw)
    P.check()
    return S, sf


@pytest.mark.parametrize("precision,m", [("fp32", m) for m in (7169, 8961, 10753, 12545, 14335, 15999)] +
                         [("fp64", m) for m in (4481, 5376, 6143)])
def test_many_rows(cuda, m, precision):
    """5 to 8 chunks per warp at 448 threads and beyond (FP64 6)."""
    A, b = _polytope(m, 4, seed=m)
    S, _ = _run(Polytope(A, b), precision=precision)
    assert np.array_equal(S, O.chr_run(A, b, np.zeros(4), 15, 3, 3, seed=5, pair_prob=0.4, resync_interval=11,
                                       precision=precision))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("m", [5, 63, 129, 321, 1283, 3841, 5375])
def test_final_slack(cuda, m, precision):
    P = Polytope(*_polytope(m, 5, seed=m))
    a, b = _run(P, precision=precision), _run(P, precision=precision, max_slots=2)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["plain", "subnormal", "huge", "small_bounds"])
@pytest.mark.parametrize("m", [150, 901, 2500, 3300])
def test_every_row_divided(cuda, m, kind, precision):
    """Two rows of zero width take half of the steps off the short cut, at each
    of the smaller thread counts; with entries whose quotients are not normal
    numbers, and with all slacks small."""
    A, b = _polytope(m, 6, seed=m)
    row = np.concatenate([np.ones(3), np.zeros(3)])
    A, b = np.vstack([A, row, -row]), np.concatenate([b, [0.0, 0.0]])
    if kind == "subnormal":
        A[5::7] *= 1e-40
    elif kind == "huge":
        A[5::7] *= 1e16
        b[5::7] *= 1e-20
    elif kind == "small_bounds":
        b = b * 1e-18
    S = Polytope(A, b)
    kw = dict(seed=5, pair_prob=0.4, resync_interval=11, precision=precision)
    got = S.run(np.zeros(6), 20, 3, 3, out_dtype="f64", sparse="dense", **kw)
    S.check()
    assert np.array_equal(got, O.chr_run(A, b, np.zeros(6), 20, 3, 3, **kw), equal_nan=True)
