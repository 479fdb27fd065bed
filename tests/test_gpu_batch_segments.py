"""Batched runs that go in several segments (GPU): at least 2^19 cells, an
interval that does not divide the run, uneven row counts, one to nine chains
(every group size of the slack kernel and a remainder).  Samples and last
states are the standalone runs', bit for bit; a captured graph replays them."""
import numpy as np
import pytest

from naja_b200 import Polytope, synth
from naja_b200.batch import Batch, Shape

pytestmark = pytest.mark.gpu

SHAPES = [Shape(256, 3, 1, 0), Shape(128, 4, 1, 0, sparse=1)]
KW = dict(seed=7, pair_prob=0.3, resync_interval=40)
NSPC, THIN = 15, 7  # 105 steps: segments of 40, 40 and 25


@pytest.fixture(scope="module")
def polys():
    base = synth.genome_shaped(n=700, d=400, density=0.08, seed_T=3, seed_u=4)
    out = [(base["A"], base["b"])]
    for v in synth.conditioned_variants(base, 2, max_reactions=25, seed=9):
        out.append((np.vstack([base["A"], v["extra_A"]]), np.concatenate([base["b"], v["extra_b"]])))
    assert len({A.shape[0] for A, _ in out}) > 1 and all(A.size >= 2 ** 19 for A, _ in out)
    return out, base["start"]


def _buffers(n, nch, d, start):
    import torch

    X = [torch.from_numpy(np.broadcast_to(start, (nch, d)).copy()).cuda() for _ in range(n)]
    outs = [torch.empty((NSPC * nch, d), dtype=torch.float64, device="cuda") for _ in range(n)]
    return X, outs, [torch.empty_like(x) for x in X]


@pytest.mark.parametrize("nch", [1, 3, 5, 9])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_segments_equal_standalone(cuda, polys, shape, nch):
    models, start = polys
    P = [Polytope(A, b) for A, b in models]
    X, outs, last = _buffers(len(P), nch, len(start), start)
    last[1] = None
    B = Batch(P)
    B.run(X, outs, NSPC, THIN, nch, shape=shape, seed_stride=5, X_finals=last, out_dtype="f64", **KW)
    B.check()
    for k, p in enumerate(P):
        xf = np.empty((nch, len(start)))
        ref = p.run(start, NSPC, THIN, nch, X_final=xf, out_dtype="f64", **dict(KW, seed=7 + 5 * k))
        assert np.array_equal(outs[k].cpu().numpy(), ref), k
        assert last[k] is None or np.array_equal(last[k].cpu().numpy(), xf), k
        assert np.array_equal(X[k].cpu().numpy(), np.broadcast_to(start, (nch, len(start))))


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_graph_of_segments_replays(cuda, polys, shape):
    import torch

    models, start = polys
    P = [Polytope(A, b) for A, b in models]
    nch = 3
    X, outs, last = _buffers(len(P), nch, len(start), start)
    B = Batch(P)
    B.run(X, outs, NSPC, THIN, nch, shape=shape, X_finals=last, out_dtype="f64", **KW)
    want = [t.clone() for t in outs + last]
    g = B.capture(X, outs, NSPC, THIN, nch, shape=shape, X_finals=last, out_dtype="f64", **KW)
    for _ in range(2):
        for t in outs + last:
            t.zero_()
        g.launch()
        g.check()
        assert all(torch.equal(a, b) for a, b in zip(outs + last, want))
    g.close()
