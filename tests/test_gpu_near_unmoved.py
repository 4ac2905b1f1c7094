"""Chains of the near / far split (rd_near.cuh) that never leave their start.  A start that
was found in a later round has the field that k_mh_init summed, and the emission test reads
that very value, in the pair-sum jumps and here: with one jump, and with electrons that
turn many first draws down, the escape probabilities agree bit for bit."""
import numpy as np
import pytest

from test_gpu_near import NM, _kw, _run, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("count", [1, 2])   # a lone diode has a kernel of its own
def test_chains_that_never_move(rg, fp64, count):
    diodes = []
    for k in range(count):
        r = np.random.default_rng(8 + k)
        n, side = 8000, 300.0
        pos = np.column_stack([r.uniform(-150, 150, n), r.uniform(-150, 150, n), r.uniform(0.6, 1.2, n)]) * NM
        kw = dict(_kw(side, side, n + 6000, V=4.0e3, max_chains=4000), mh_jumps=1, seed=90 + k, time_step=1.0e-15)
        diodes.append((kw, pos))
    fast, slow = (_run(rg, diodes, 1, atom, fp64=fp64) for atom in (False, True))
    assert fast[0][1]["chains"] > 500
    _same(fast, slow)
