"""Calls from several threads on streams of their own, whose launches of one
kernel differ in shared memory (GPU): every call gives what it gives alone."""
import threading

import numpy as np
import pytest

from naja_b200 import Polytope
from naja_b200 import validate as nv
from naja_b200.batch import Batch, Shape

pytestmark = pytest.mark.gpu


def _polytope(m, d):
    rng = np.random.default_rng(d)
    half = rng.standard_normal((m // 2, d))
    return Polytope(np.concatenate([half, -half]), 10.0 ** rng.uniform(0.0, 2.0, m))


def _together(works, times):
    """Each work (a call that returns arrays or tensors) alone, then all at once, `times` times."""
    import torch

    def values(out):
        return [t.cpu().numpy().copy() if hasattr(t, "cpu") else np.array(t) for t in out]

    want, errors = [], []
    for w in works:
        out = w()
        torch.cuda.synchronize()
        want.append(values(out))

    def loop(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(times):
                    out = works[k]()
                torch.cuda.current_stream().synchronize()
                assert all(np.array_equal(a, b) for a, b in zip(values(out), want[k], strict=True))
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(works))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors[:2]


@pytest.mark.parametrize("sparse", ["dense", "columns"])
def test_runs(cuda, sparse):
    import torch

    def work(d):
        P = _polytope(200, d)
        X = torch.zeros((2, d), dtype=torch.float64, device="cuda")
        out = torch.empty((8, d), device="cuda")
        return lambda: [P.run(X, 4, 2, out=out, seed=1, sparse=sparse)]

    _together([work(d) for d in (20, 2500, 40, 3000)], 300)


def test_batches(cuda):
    import torch

    def work(m, d, sparse):
        P = [_polytope(m, d) for _ in range(2)]
        B = Batch(P)
        X = [torch.zeros((2, d), dtype=torch.float64, device="cuda") for _ in P]
        outs = [torch.empty((8, d), device="cuda") for _ in P]
        shape = Shape(128, 3, 1, 0, sparse)

        def run():
            B.run(X, outs, 4, 2, 2, shape=shape, seed=1, resync_interval=5)
            return outs

        return run

    _together([work(400, 1400, 0), work(300, 2500, 0), work(400, 1350, 0)], 100)


def test_validation(cuda):
    rng = np.random.default_rng(0)

    def work(spc, chains, dim):
        S = rng.standard_normal((spc * chains, dim)).astype(np.float32)
        return lambda: nv.ess_rhat(S, chains)

    _together([work(40, 2, 3), work(9000, 2, 2), work(60, 300, 9), work(20000, 1, 1)], 100)
