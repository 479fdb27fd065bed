"""Which step kernel and launch shape a run takes, and what is refused (GPU)."""
import numpy as np
import pytest

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
