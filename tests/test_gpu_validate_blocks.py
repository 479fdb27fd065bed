"""ESS and R-hat around the edges of the lag blocks, the series slices and the
coordinate groups (GPU), against the CPU oracle; ESS rtol 1e-4 and R-hat 1e-9
as in test_gpu_validate.py, whose reasons hold here."""
import numpy as np
import pytest

import oracle.oracle as O
from naja_b200 import validate as nv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("spc,nchains,dim", [(4, 1, 1), (5, 3, 9), (63, 2, 7), (66, 1, 8), (130, 2, 33), (1000, 1, 3),
                                             (4000, 2, 9), (13000, 1, 2), (26000, 1, 1), (49152, 1, 1)])
def test_edges(cuda, spc, nchains, dim, layout):
    rng = np.random.default_rng(spc)
    x = rng.standard_normal((spc, nchains, dim))
    rho = 0.97 if spc >= 1000 else 0.5
    for t in range(1, spc):
        x[t] = rho * x[t - 1] + np.sqrt(1 - rho * rho) * x[t]
    S = np.ascontiguousarray(x.reshape(spc * nchains, dim) + 3.0).astype(np.float32)
    ess, rhat = nv.ess_rhat(S, nchains, layout=layout)
    assert np.allclose(ess, O.ess(S, nchains, layout), rtol=1e-4)
    assert np.allclose(rhat, O.split_rhat(S, nchains, layout), rtol=1e-9)
