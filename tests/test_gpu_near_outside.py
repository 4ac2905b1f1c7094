"""Proposals off the emitter.  A step size above its clamp, which only a checkpoint can bring,
reflects a proposal once and may leave it outside, where no panel's expansion holds: the
chains of the near / far split are still those of the pair-sum jumps."""
import struct

import numpy as np
import pytest

from test_gpu_near import NM, _electrons, _kw, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
@pytest.mark.parametrize("std", [0.3, 0.9, 3.0])
def test_step_size_from_a_checkpoint(rg, prec, std):
    kw = dict(_kw(300.0, 300.0, 9000, max_chains=4000), mh_jumps=4, time_step=1.0e-15)
    pos = _electrons(1500, 300.0, 300.0, 1000.0, 21)
    res = []
    for atom in (False, True):
        with rg.Engine(precision=getattr(rg, prec), max_diodes=1, particle_capacity=9100, chain_capacity=9100,
                       quad_capacity=rg.supply_points(**kw) + 64) as eng:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            state = bytearray(d.save_state())
            at = bytes(state[:2048]).index(struct.pack("<d", d.counters()["MH_std"]))
            state[at:at + 8] = struct.pack("<d", std)
            d.load_state(bytes(state))
            if atom:
                d.add_particle((0.0, 0.0, 900.0 * NM), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            assert d.counters()["MH_std"] == std
            eng.run(1, 1)
            res.append((d.particles(), d.counters()))
    assert res[0][1]["chains"] > 500
    _same(res[:1], res[1:])
