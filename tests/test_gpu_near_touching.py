"""FP64 chains of the near / far split (rd_near.cuh) with electrons 1e-6 to 1e-4 nm above
the cathode under supply nodes.  There the l^2 of the reference's r + l^2 and the last bits
of an FP32 pair of coordinates show in an electron's term, which the estimate of the field
leaves out: its bound has to carry them.  The chains are those of the pair-sum jumps."""
import numpy as np
import pytest

from test_gpu_near import NM, _electrons, _kw, _run, _same
from test_gpu_near_nodes import nodes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("low,high", [(1.0e-6, 1.0e-5), (1.0e-5, 1.0e-4), (1.0e-4, 1.0e-3)])
def test_electrons_touching_the_cathode(rg, n, low, high):
    side = 300.0
    kw = _kw(side, side, 6000, max_chains=1500)
    x, y = nodes(rg, kw, n, 5)
    r = np.random.default_rng(6)
    pos = np.vstack([np.column_stack([x, y, np.exp(r.uniform(np.log(low), np.log(high), n))]) * NM,
                     _electrons(200, side, side, 1000.0, 7)])
    fast, slow = (_run(rg, [(kw, pos)], 1, atom, fp64=True) for atom in (False, True))
    assert fast[0][1]["chains"] > 100
    _same(fast, slow)
