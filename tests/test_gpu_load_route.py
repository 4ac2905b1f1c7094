"""A checkpoint replaces the whole state of a diode, so a diode that held an atom (and took
the pair-sum jumps for it) and then loads a state of electrons only takes the near / far
split again, with the same chains as a diode that never held one."""
import numpy as np
import pytest

import test_gpu_tip_near as tip
from test_gpu_near import NM, _electrons, _kw, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("geometry", ["planar", "tip"])
def test_electrons_after_an_atom(rg, geometry):
    if geometry == "tip":
        kw, pos = tip._case("close")
        kw = dict(kw, geometry=rg.GEOM_TIP)
    else:
        kw, pos = _kw(400.0, 400.0, 6000), _electrons(900, 400.0, 400.0, 1000.0, 9)
    cap = kw["capacity"] + 64
    out = []
    for atom in (False, True):
        with rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=cap, chain_capacity=cap,
                       quad_capacity=rg.supply_points(**kw) + 64) as eng:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            state = d.save_state()
            if atom:
                d.add_particle((0.0, 0.0, 900.0 * NM), species=rg.ATOM, step=0)
                eng.run(1, 1)
                d.load_state(state)
            eng.run(1, 2)
            out.append((d.particles(), d.counters(), eng.last_run_stats()[1]))
    _same([out[0][:2]], [out[1][:2]])
    assert out[0][2] == out[1][2]
