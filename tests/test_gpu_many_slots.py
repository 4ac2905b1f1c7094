"""An engine with more diode slots than a launch grid has rows (65535): a tip emits and steps
in it as in a small one."""
import numpy as np
import pytest

import test_gpu_tip_near as tip

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
def test_tip_in_a_wide_engine(rg, prec):
    kw, pos = tip._case("tile-edge")
    kw = dict(kw, geometry=rg.GEOM_TIP, max_chains=1000)
    res = []
    for slots in (1, 65600):
        with rg.Engine(precision=getattr(rg, prec), max_diodes=slots, particle_capacity=16000, chain_capacity=4096,
                       quad_capacity=10064) as eng:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            eng.run(1, 2)
            res.append((d.particles(), d.counters()))
    assert res[0][1]["chains"] > 0
    tip._same(res[:1], res[1:])
