"""The network's GEMM at the edges of each tile width (GPU): M on both sides of
64 and 128, N on both sides of 16, 32, 64 and 128 columns, K past the ring's
depth, every output.  FP32 accumulation: K 2^-24 of the row's absolute sum
(K additions of half an ulp each)."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 16, 64), (65, 17, 72), (63, 512, 1100), (128, 9500, 64), (64, 9480, 136),
                                   (1200, 1050, 200), (4736, 150, 65)])
def test_gemm_tiles(cuda, M, N, K):
    import torch

    from naja_b200._lib import GemmEpilogue, check, load

    rng = np.random.default_rng(M + N)
    pad = lambda n: (n + 7) // 8 * 8  # noqa: E731
    A, B = torch.zeros((M, pad(K)), dtype=torch.bfloat16), torch.zeros((N, pad(K)), dtype=torch.bfloat16)
    A[:, :K] = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32))
    B[:, :K] = torch.from_numpy(rng.standard_normal((N, K)).astype(np.float32))
    bias = torch.from_numpy(rng.standard_normal(N).astype(np.float32)).cuda()
    A, B = A.cuda(), B.cuda()
    c = torch.full((M, N + 1), 7.0, device="cuda")
    act = torch.full((M, pad(N)), 3.0, dtype=torch.bfloat16, device="cuda")
    act_t = torch.full((N, pad(M)), 3.0, dtype=torch.bfloat16, device="cuda")
    lib = load()
    e = GemmEpilogue(bias.data_ptr(), c.data_ptr(), N + 1, 0, act.data_ptr(), pad(N), act_t.data_ptr(), pad(M), 1)
    check(lib.naja_gemm_bf16(M, N, K, A.data_ptr(), pad(K), B.data_ptr(), pad(K), C.byref(e), None))
    check(lib.naja_mlp_check(None))
    a64, b64 = A[:, :K].double(), B[:, :K].double()
    ref = a64 @ b64.T + bias.double()
    tol = (K + 1) * 2.0 ** -24 * (a64.abs() @ b64.abs().T + bias.double().abs())
    assert bool(((c[:, :N].double() - ref).abs() <= tol).all()) and bool((c[:, N] == 7.0).all())
    g = act[:, :N].float().cpu().numpy()
    assert np.allclose(g, MO.bf16(MO.gelu(c[:, :N].cpu().numpy().astype(np.float64))), rtol=2 ** -7, atol=1e-6)
    assert np.array_equal(act_t[:, :M].float().cpu().numpy(), g.T)
    assert bool((act[:, N:] == 3.0).all()) and bool((act_t[:, M:] == 3.0).all())


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (32, 64), (65, 100), (3, 1000)])
def test_cast_tiles(cuda, rows, cols):
    import torch

    from naja_b200._lib import check, load

    src = torch.randn((rows, cols + 2), device="cuda")
    dst = torch.full((rows, cols + 1), 5.0, dtype=torch.bfloat16, device="cuda")
    dst_t = torch.full((cols, rows + 3), 5.0, dtype=torch.bfloat16, device="cuda")
    check(load().naja_cast_bf16(rows, cols, src.data_ptr(), cols + 2, dst.data_ptr(), cols + 1, dst_t.data_ptr(), rows + 3,
                                None))
    want = src[:, :cols].to(torch.bfloat16)
    assert torch.equal(dst[:, :cols], want) and torch.equal(dst_t[:, :rows], want.t())
    assert bool((dst[:, cols:] == 5.0).all()) and bool((dst_t[:, rows:] == 5.0).all())
