"""The rounding network under a current stream that is not the default one:
its copies and its kernels stay in one order."""
import contextlib
import types

import numpy as np
import pytest

from naja_b200 import learned


def test_copies_and_kernels_share_a_stream(monkeypatch):
    """With stand-ins for the library and the streams (CPU): the current stream
    at every kernel launch is the kernel's, and waits for and is waited for by
    the caller's."""
    torch = pytest.importorskip("torch")
    side = types.SimpleNamespace(cuda_stream=7)
    own = types.SimpleNamespace(cuda_stream=0)
    log, current = [], [side]
    side.wait_stream = lambda s: log.append(("side waits", s.cuda_stream))
    own.wait_stream = lambda s: log.append(("own waits", s.cuda_stream))

    @contextlib.contextmanager
    def use(s):
        current.append(s)
        yield
        current.pop()

    class Lib:
        def __getattr__(self, name):
            return lambda *a: log.append((name, a[-1], current[-1].cuda_stream)) or 0

    monkeypatch.setattr(learned, "_current_handle", lambda torch, device: current[-1].cuda_stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: current[-1])
    monkeypatch.setattr(torch.cuda, "default_stream", lambda device=None: own)
    monkeypatch.setattr(torch.cuda, "stream", use)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **kw: empty(*a, **kw))
    monkeypatch.setattr(learned, "load", Lib)
    monkeypatch.setattr(learned, "check", lambda st: None)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, s: log.append(("record", s.cuda_stream)))

    net = learned.RoundingNet((6, 4, 3), device="cpu")
    X, T = np.ones((2, 6), np.float32), np.ones((2, 3), np.float32)
    net.train_step(X, T)
    net.predict(X)
    net.restore(net.snapshot())
    kernels = [e for e in log if e[0].startswith("naja_")]
    assert {e[0] for e in kernels} >= {"naja_gemm_bf16", "naja_mse_grad", "naja_adam", "naja_cast_bf16"}
    assert all(stream == cur for _, stream, cur in kernels)
    assert log[0] == ("own waits", 7) and log[-1] == ("side waits", 0)
    assert log.count(("own waits", 7)) == log.count(("side waits", 0))
    assert log.count(("record", 7)) == 1 + 2 * 2  # the prediction, a snapshot of two layers


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["host", "device"])
def test_side_stream_gradients(cuda, where):
    """Gradients of alternating batches under a side stream are the default stream's, bit for bit."""
    import torch

    rng = np.random.default_rng(0)
    dims, B = (640, 256, 20000), 48
    batches = [(rng.standard_normal((B, dims[0]), dtype=np.float32), rng.standard_normal((B, dims[-1]), dtype=np.float32))
               for _ in range(3)]
    if where == "device":
        batches = [(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()) for X, T in batches]

    def grads():
        net = learned.RoundingNet(dims, seed=1)
        out = []
        for X, T in batches * 2:
            net.gradients(X, T)
            out += [t.clone() for L in net.layers for t in (L.gW, L.gb)]
        out.append(net.predict(batches[0][0]))
        return out

    want = grads()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        got = grads()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want, strict=True))
