"""Which step kernel and launch shape a run takes, and what is refused (GPU)."""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import Polytope
from naja_b200._lib import InvalidArgument

pytestmark = pytest.mark.gpu


def _dense(m, d, seed=0):
    """m dense rows around the origin, bounded in every direction."""
    rng = np.random.default_rng(seed)
    half = rng.standard_normal(((m + 1) // 2, d))
    return np.concatenate([half, -half])[:m], 10.0 ** rng.uniform(0.0, 2.0, m)


@pytest.mark.parametrize("tpb", [31, 96, 192, 448, 992])
def test_forced_thread_counts_are_the_references(cuda, tpb):
    """Counts that only the library's own choice uses are refused when forced."""
    P = Polytope(*_dense(600, 5))
    with pytest.raises(InvalidArgument, match="Invalid threads per block"):
        P.kernel_choice(10, 1, 2, tpb=tpb)
    with pytest.raises(InvalidArgument, match="Invalid threads per block"):
        P.run(np.zeros(5), 10, 1, 2, tpb=tpb)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_general_kernel_runs_uniform_chunks(cuda, precision):
    """Runs that divide every row (k-sparse steps, an infinite bound) on 14
    warps where those hold the rows in as many chunks as 16."""
    A, b = _dense(5200, 4)
    P = Polytope(A, b)
    kw = dict(precision=precision, sparse="dense")
    assert P.kernel_choice(10, 1, 2, ksparse_prob=0.2, **kw)["threads"] == 448
    b = b.copy()
    b[3] = np.inf
    assert Polytope(A, b).kernel_choice(10, 1, 2, **kw)["threads"] == 448


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("kw", [dict(ksparse_prob=0.3, ksparse_k=3), dict(infinite=True), dict(infinite=True, tpb=1024)], ids=str)
@pytest.mark.parametrize("m", [6, 8, 132, 642, 1284, 5200])
def test_general_kernel_against_the_oracle(cuda, m, kw, precision):
    """Bit for bit (both tiers give the oracle's samples exactly), row counts
    that are and are not multiples of a lane's rows."""
    kw = dict(kw)
    A, b = _dense(m, 5, seed=m)
    if kw.pop("infinite", False):
        b[1] = np.inf
    run = dict(seed=5, pair_prob=0.4, resync_interval=11, precision=precision)
    P = Polytope(A, b)
    dt = np.float64 if precision == "fp64" else np.float32
    slack, sf = np.empty((3, m), dt), np.empty((3, m), dt)
    got = P.run(np.zeros(5), 25, 3, 3, out_dtype="f64", sparse="dense", slack_final=slack, **run, **kw)
    P.check()
    tpb = kw.pop("tpb", None)
    assert np.array_equal(got, O.chr_run(A, b, np.zeros(5), 25, 3, 3, **run, **kw), equal_nan=True)
    # with other threads, columns straight from global memory
    P.run(np.zeros(5), 25, 3, 3, out_dtype="f64", sparse="dense", slack_final=sf, max_slots=2, tpb=tpb or 256, **run, **kw)
    P.check()
    assert np.array_equal(slack, sf, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("m,pair", [(120, 0.4), (700, 1.0), (5200, 0.4)])
def test_rows_of_zero_width(cuda, m, pair, precision):
    """Steps that divide every row among screened ones, bit for bit: two
    opposite rows that leave half of the coordinates no room."""
    A, b = _dense(m, 6, seed=m)
    row = np.concatenate([np.ones(3), np.zeros(3)])
    A, b = np.vstack([A, row, -row]), np.concatenate([b, [0.0, 0.0]])
    run = dict(seed=5, pair_prob=pair, resync_interval=11, precision=precision)
    P = Polytope(A, b)
    got = P.run(np.zeros(6), 25, 4, 3, out_dtype="f64", sparse="dense", **run)
    P.check()
    assert np.array_equal(got, O.chr_run(A, b, np.zeros(6), 25, 4, 3, **run), equal_nan=True)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_resident_columns_only_where_the_chains_fit(cuda, precision):
    """The unit cube of d = 400: all columns in shared memory for few chains,
    a ring of them where the copies would keep chains waiting; same samples."""
    d = 400
    P = Polytope(np.vstack([np.eye(d), -np.eye(d)]), np.concatenate([np.ones(d), np.zeros(d)]))
    kw = dict(seed=5, pair_prob=0.3, precision=precision)
    few, many = P.kernel_choice(4, 8, 3, **kw), P.kernel_choice(4, 8, 600, **kw)
    assert few["kernel"] == many["kernel"] == "columns"
    assert few["smem"] > 100 << 10 and many["smem"] < 40 << 10, (few, many)
    a = P.run(np.full(d, 0.5), 4, 8, 3, **kw)
    b = P.run(np.full(d, 0.5), 4, 8, 600, **kw)
    P.check()
    assert np.array_equal(a.reshape(4, 3, d), b.reshape(4, 600, d)[:, :3])
