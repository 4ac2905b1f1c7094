"""FP64 chains of the near / far split (rd_near.cuh) on wide emitters, with electrons just
above the cathode beside the supply panels' Gauss-Legendre nodes: half an ulp of an FP32
coordinate (up to 5e-4 nm at 10 um) is then a visible part of the distance, so the panels'
near and far parts have to be taken at the nodes themselves.  The chains are those of the
pair-sum jumps (a diode that once held an atom keeps those)."""
import numpy as np
import pytest

from test_gpu_near import NM, _kw, _run, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def nodes(rg, kw, n, seed):
    """n of the emitter's supply nodes (nm), in different panels where there are enough."""
    q = int(round(np.sqrt(rg.supply_points(**kw))))
    panels, r = q // 4, np.random.default_rng(seed)
    t = np.polynomial.legendre.leggauss(4)[0]
    lx, ly = (v / NM for v in kw["emitter_dim"])
    k = r.permutation(panels * panels)[:n] if n <= panels * panels else r.integers(0, panels * panels, n)
    gx, gy = t[r.integers(0, 4, n)], t[r.integers(0, 4, n)]
    x = -lx / 2 + lx / panels * (k % panels + 0.5 * (1.0 + gx))
    y = -ly / 2 + ly / panels * (k // panels + 0.5 * (1.0 + gy))
    return x, y


@pytest.mark.parametrize("side,n", [(2000.0, 8000), (8000.0, 20000), (20000.0, 20000)])
@pytest.mark.parametrize("low,high", [(0.05, 0.5), (0.5, 1.5)])
def test_low_electrons_beside_nodes(rg, side, n, low, high):
    kw = _kw(side, side, n + 6000, max_chains=12000)
    x, y = nodes(rg, kw, n, 3)
    r = np.random.default_rng(4)
    z = r.uniform(low, high, n)
    ang, off = r.uniform(0.0, 2.0 * np.pi, n), 0.5 * z
    pos = np.column_stack([x + off * np.cos(ang), y + off * np.sin(ang), z]) * NM
    fast, slow = (_run(rg, [(kw, pos)], 1, atom, fp64=True) for atom in (False, True))
    assert fast[0][1]["chains"] == 12000
    _same(fast, slow)
