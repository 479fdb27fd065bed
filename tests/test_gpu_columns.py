"""The private-rows compressed-column kernel against the CPU oracle, bit for bit (GPU).

Both tiers give the oracle's samples exactly, so the tolerance is zero:
column lengths around each count of entries per lane and of row warps, rows
of uneven weight, columns kept in shared memory and staged ones, and the
inputs that take a step off its short cut.
"""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import Polytope

pytestmark = pytest.mark.gpu


def _polytope(m, d, per_col, seed, heavy=0):
    """`per_col` nonzeros in every column, `heavy` more in the first rows of column 0, both signs."""
    rng = np.random.default_rng(seed)
    A = np.zeros((m, d))
    for j in range(d):
        r = rng.choice(m, size=per_col, replace=False)
        A[r, j] = rng.standard_normal(per_col)
        A[r[0], j], A[r[1], j] = 1.0, -1.0
    A[:heavy, 0] = rng.standard_normal(heavy)
    return A, 10.0 ** rng.uniform(0.0, 2.0, m), np.zeros(d)


def _same(A, b, x0, precision, nspc=25, thin=4, nchains=3, seed=5, **kw):
    P = Polytope(A, b)
    kw = dict(dict(pair_prob=0.4, resync_interval=13), **kw)
    got = P.run(x0, nspc, thin, nchains, seed=seed, precision=precision, out_dtype="f64", sparse="columns", **kw)
    P.check()
    ref = O.chr_run(A, b, x0, nspc, thin, nchains, seed=seed, precision=precision,
                    **{k: v for k, v in kw.items() if k not in ("max_slots", "tpb")})
    assert np.array_equal(got, ref, equal_nan=True), np.nanmax(np.abs(got - ref))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("per_col", [2, 31, 33, 65, 97, 129, 193, 257, 520, 700])
def test_column_lengths(cuda, per_col, precision):
    _same(*_polytope(max(40, 4 * per_col), 6, per_col, seed=per_col), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kw", [dict(tpb=32), dict(tpb=64), dict(tpb=128), dict(tpb=256), dict(max_slots=3),
                                dict(max_slots=8, pair_prob=1.0), dict(resync_interval=0, pair_prob=0.0)])
def test_launch_shapes(cuda, kw, precision):
    _same(*_polytope(333, 9, 40, seed=1), precision, **kw)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("heavy", [60, 300, 900])
def test_uneven_rows(cuda, heavy, precision):
    """A column with up to 900 entries among short ones (the longest takes the other kernel)."""
    _same(*_polytope(1000, 12, 6, seed=heavy, heavy=heavy), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", ["vertex", "wide_pairs", "huge"])
def test_off_the_short_cut(cuda, case, precision):
    A, b, x0 = _polytope(120, 6, 12, seed=2)
    kw = {}
    if case == "vertex":  # every slack of the start is zero
        A, b, x0 = np.vstack([np.eye(6), -np.eye(6)]), np.concatenate([np.ones(6), np.zeros(6)]), np.zeros(6)
    elif case == "wide_pairs":
        kw.update(pair_mode=2, pairs=([0, 2], [1, 3], [0.6, 5.0], [0.8, 0.25]))
    else:
        A[7] *= 1e20
        b[7] *= 1e20
    _same(A, b, x0, precision, **kw)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_unbounded_coordinate(cuda, precision):
    """An infinite step leaves the rows it does not touch alone (the oracle's
    inf * 0 makes them NaN), so the other compressed-column kernel is the reference."""
    A, b, x0 = _polytope(120, 6, 12, seed=2)
    A[:, 3] = -np.abs(A[:, 3])  # no row ends coordinate 3 upwards
    P = Polytope(A, b)
    kw = dict(seed=5, pair_prob=0.4, resync_interval=13, precision=precision, out_dtype="f64", sparse="columns")
    got, ref = P.run(x0, 25, 4, 3, **kw), P.run(x0, 25, 4, 3, tpb=512, **kw)
    assert np.isinf(ref).any() and np.array_equal(got, ref, equal_nan=True)
