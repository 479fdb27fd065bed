"""ESS and R-hat over every length of lag block, and R-hat with more half-chains
than a CTA keeps the means of (GPU), against the CPU oracle; ESS rtol 1e-4 and
R-hat 1e-9 as in test_gpu_validate.py, whose reasons hold here."""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import validate as nv

pytestmark = pytest.mark.gpu


def _series(spc, nchains, dim, rho, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((spc, nchains, dim))
    for t in range(1, spc):
        x[t] = rho * x[t - 1] + np.sqrt(1 - rho * rho) * x[t]
    return np.ascontiguousarray(x.reshape(spc * nchains, dim) + 3.0).astype(np.float32)


@pytest.mark.parametrize("rho", [0.0, 0.9, 0.99, 0.997, 0.9995])
def test_lag_blocks(cuda, rho):
    """Series that stop after 1 lag to some 2,000, so in blocks of 64 to 512 lags."""
    S = _series(8000, 2, 3, rho, seed=11)
    ess, rhat = nv.ess_rhat(S, 2)
    assert np.allclose(ess, O.ess(S, 2, 1), rtol=1e-4)
    assert np.allclose(rhat, O.split_rhat(S, 2, 1), rtol=1e-9)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("spc,nchains,dim", [(9, 1, 1), (21, 17, 2), (300, 5, 8), (64, 16, 9), (9, 1500, 9), (6, 5000, 1)])
def test_rhat_half_chains(cuda, spc, nchains, dim, layout):
    S = _series(spc, nchains, dim, 0.3, seed=spc)
    _, rhat = nv.ess_rhat(S, nchains, layout=layout, ess=False)
    assert np.allclose(rhat, O.split_rhat(S, nchains, layout), rtol=1e-9)
