"""The network's GEMM at each tile width with one and with several tiles per SM
(GPU), ragged in every dimension.  FP32 accumulation: K 2^-24 of the row's
absolute sum (K additions of half an ulp each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(33, 500, 1100), (300, 530, 1100), (1300, 530, 1100), (2100, 530, 900), (2100, 1100, 900),
                                   (60, 4801, 700), (33, 9601, 700), (1900, 2100, 300)])
def test_gemm_widths(cuda, M, N, K):
    import ctypes as C

    import torch

    from naja_b200._lib import GemmEpilogue, check, load

    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    ld = (K + 7) // 8 * 8
    A = torch.randn((M, ld), generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn((N, ld), generator=g, device="cuda").to(torch.bfloat16)
    c = torch.full((M, N + 1), 7.0, device="cuda")
    lib = load()
    e = GemmEpilogue(None, c.data_ptr(), N + 1, 0, None, 0, None, 0, 0)
    check(lib.naja_gemm_bf16(M, N, K, A.data_ptr(), ld, B.data_ptr(), ld, C.byref(e), None))
    check(lib.naja_mlp_check(None))
    a, b = A[:, :K].double(), B[:, :K].double()
    tol = (K + 1) * 2.0 ** -24 * (a.abs() @ b.abs().T)
    assert bool(((c[:, :N].double() - a @ b.T).abs() <= tol).all()) and bool((c[:, N] == 7.0).all())
