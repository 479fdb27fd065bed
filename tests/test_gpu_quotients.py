"""The screened kernel's branch-free arithmetic (GPU): reciprocals and quotients
equal to the IEEE ones where a certain step uses them, and the error of the
FP64 estimates.  The bounds are those that chr_screen.cuh's derivation states:
2^-19 for an operand of 21 significant bits; the estimate drops an operand's
low word, 2^-20 relative, so 2^-18 for any."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    if not Path(NVCC).exists():
        pytest.skip("no nvcc")
    so = tmp_path_factory.mktemp("quotients") / "quotients.so"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", str(ROOT / "include"), str(ROOT / "tests" / "cuda" / "quotients.cu"),
                    "-o", str(so)], check=True, capture_output=True, text=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("e", [-120, -60, -1, 0, 1, 60, 119])
def test_reciprocals(lib, e):
    import torch

    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert lib.check_reciprocals(e, C.c_void_p(bad.data_ptr())) == 0
    assert int(bad) == 0


@pytest.mark.parametrize("seed", [0, 1])
def test_quotients(lib, seed):
    import torch

    n = torch.zeros(2, dtype=torch.int64, device="cuda")
    assert lib.check_quotients(seed, C.c_void_p(n.data_ptr()), C.c_void_p(n.data_ptr() + 8)) == 0
    assert int(n[0]) == 0 and int(n[1]) > 1 << 25


@pytest.mark.parametrize("e", [-500, -42, 0, 1, 300])
def test_estimates(lib, e):
    import torch

    worst = torch.zeros(2, dtype=torch.float64, device="cuda")
    assert lib.check_estimates(e, C.c_void_p(worst.data_ptr()), C.c_void_p(worst.data_ptr() + 8)) == 0
    assert 0.0 < float(worst[0]) < 2.0 ** -19 and float(worst[1]) < 2.0 ** -18
