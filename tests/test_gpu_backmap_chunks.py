"""The tensor-core backmap over more samples than it maps at a time (GPU).
Tolerances as in test_gpu_backmap.py: 2^-15 (BF16X3) and 2^-17 (TF32X3) of
sum_k |T_ik y_k| + |shift_i|."""
import numpy as np
import pytest

from naja_b200 import backmap

pytestmark = pytest.mark.gpu

TOL = {"bf16x3": 2.0 ** -15, "tf32x3": 2.0 ** -17}


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("mode,N", [("tf32x3", 25_013), ("bf16x3", 45_001)])
def test_chunks(cuda, mode, N, dtype):
    """d = 1,501: a chunk is at most 9,472 (BF16X3 18,944) samples."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    n, d = 70, 1501
    T = torch.randn((n, d), generator=g, device="cuda", dtype=torch.float64)
    shift = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    scale = 10.0 ** (4.0 * torch.rand((1, d), generator=g, device="cuda") - 2.0)
    Y = (torch.randn((N, d), generator=g, device="cuda") * scale).to(getattr(torch, dtype))
    V = torch.full((N + 1, n), -3.0, dtype=torch.float64, device="cuda")
    backmap(T, shift, Y, mode=mode, out=V[:N])
    ref = Y.double() @ T.T + shift
    lim = Y.double().abs() @ T.T.abs() + shift.abs()
    assert float(((V[:N] - ref).abs() / lim).max()) <= TOL[mode]
    assert bool((V[N] == -3.0).all())
    # every row as a call of its own sample block gives it
    part = torch.empty((300, n), dtype=torch.float64, device="cuda")
    for r in (0, 9_300, 18_900, N - 300):
        backmap(T, shift, Y[r:r + 300].contiguous(), mode=mode, out=part)
        assert torch.equal(V[r:r + 300], part), r
