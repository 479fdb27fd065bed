"""The screened dense step kernel against the CPU oracle, bit for bit (GPU).

Both tiers give the oracle's samples exactly, so the tolerance is zero: row
counts on and around the edges of its 128-row (FP64 64-row) chunks and of its
automatic thread counts, and the inputs that take a step off its short cut
(repeated rows that tie for an extreme, slacks of zero, slacks below its
threshold, wide pair coefficients) or the run off the kernel (entries or
bounds beyond its range).
"""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import Polytope

pytestmark = pytest.mark.gpu


def _polytope(m, d, seed, scale=1.0):
    """Dense rows around the origin, bounded in every direction; some rows twice."""
    rng = np.random.default_rng(seed)
    half = rng.standard_normal(((m + 1) // 2, d))
    A = np.concatenate([half, -half])[:m] if m > 1 else half
    b = scale * 10.0 ** rng.uniform(0.0, 2.0, m)
    k = m // 8
    A[m - k:], b[m - k:] = A[:k], b[:k]
    return A, b, np.zeros(d)


def _same(A, b, x0, precision, nspc=25, thin=3, nchains=3, **kw):
    P = Polytope(A, b)
    sf = np.empty((nchains, P.m), dtype=np.float64 if precision == "fp64" else np.float32)
    got = P.run(x0, nspc, thin, nchains, seed=5, precision=precision, out_dtype="f64", sparse="dense",
                slack_final=sf, **kw)
    P.check()
    ref = O.chr_run(A, b, x0, nspc, thin, nchains, seed=5, precision=precision,
                    **{k: v for k, v in kw.items() if k != "max_slots"})
    assert np.array_equal(got, ref, equal_nan=True), np.nanmax(np.abs(got - ref))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("m", [6, 63, 65, 127, 129, 320, 321, 641, 1279, 1281, 2561, 3841, 5377])
def test_row_counts(cuda, m, precision):
    A, b, x0 = _polytope(m, 5, seed=m)
    _same(A, b, x0, precision, pair_prob=0.4, resync_interval=11)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", ["vertex", "face", "tiny", "wide_pairs", "unbounded", "three_slots"])
def test_off_the_short_cut(cuda, case, precision):
    A, b, x0 = _polytope(150, 6, seed=9)
    kw = dict(pair_prob=0.4)
    if case == "vertex":  # every slack of the start is zero
        A, b, x0 = np.vstack([np.eye(6), -np.eye(6)]), np.concatenate([np.ones(6), np.zeros(6)]), np.zeros(6)
    elif case == "face":  # two opposite rows of zero width that half the coordinates do not touch
        row = np.concatenate([np.ones(3), np.zeros(3)])
        A, b = np.vstack([A, row, -row]), np.concatenate([b, [0.0, 0.0]])
    elif case == "tiny":
        A, b, x0 = _polytope(150, 6, seed=9, scale=1e-15)
    elif case == "wide_pairs":
        kw.update(pair_mode=2, pairs=([0, 2], [1, 3], [0.6, 5.0], [0.8, 0.25]))
    elif case == "unbounded":  # no row ends the chord upwards
        A = -np.abs(A)
    elif case == "three_slots":
        kw.update(max_slots=3)
    _same(A, b, x0, precision, **kw)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", ["entries", "bounds"])
def test_out_of_range_polytopes(cuda, case, precision):
    """Entries above 2^58 and infinite bounds take the kernel that divides every row."""
    A, b, x0 = _polytope(200, 4, seed=3)
    if case == "entries":
        A[7] *= 1e20
        b[7] *= 1e20
    else:
        b[::5] = np.inf
    _same(A, b, x0, precision, pair_prob=0.3)
