"""Pair-sum jumps of planar diodes and of tips in one engine.  The two kernels lay the partial
sums of their work items out differently in one scratch, so they must not run at the same
time: the emission of every diode in such a mix is that of the diode alone, bit for bit, at
any number of launches per planar jump."""
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


def _emit(rg, diodes, prec, parts):
    cap = sum(kw["capacity"] + 64 for kw, _, _ in diodes)
    quad = sum(rg.supply_points(**kw) + 64 for kw, _, _ in diodes)
    with rg.Engine(precision=prec, max_diodes=len(diodes), particle_capacity=cap, chain_capacity=cap,
                   quad_capacity=quad, chunk_min=128, chunk_count_max=32) as eng:
        if parts:
            eng.set_mh_launch(parts, -1)
        out = []
        for kw, pos, atom in diodes:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            if atom:
                d.add_particle((0.0, 0.0, 900.0 * NM), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            out.append(d)
        for step in (1, 2, 3):
            eng.do_emission(step)
        return [(d.particles(), d.counters()) for d in out]


@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
@pytest.mark.parametrize("near", [False, True])   # with a diode of the near / far split beside them
@pytest.mark.parametrize("parts", [0, 4])
def test_planar_and_tip_pair_sums_in_one_engine(rg, prec, near, parts):
    n = 700 if prec == "PREC_FP64" else 3000
    diodes = []
    for k in range(2):   # tips that take the pair sums (in FP32 they once held an atom)
        dims = tip._tip(250.0, 1000.0)
        kw = dict(tip._kw(dims, n + 3000, 3000.0, max_chains=500), geometry=rg.GEOM_TIP, seed=50 + k, mh_jumps=30)
        diodes.append((kw, tip._cloud(dims, n, k, 4), True))
    for k in range(3):   # planar diodes with a longer image series
        kw = dict(_kw(300.0, 300.0, n + 3000, max_chains=500), N_ic_max=1, seed=60 + k, mh_jumps=30)
        diodes.append((kw, _electrons(n, 300.0, 300.0, 1000.0, k), False))
    if near:
        diodes.insert(2, (dict(_kw(300.0, 300.0, n + 3000, max_chains=500), seed=70, mh_jumps=30),
                          _electrons(n, 300.0, 300.0, 1000.0, 9), False))
    prec = getattr(rg, prec)
    mix = _emit(rg, diodes, prec, parts)
    for d, m in zip(diodes, mix):
        alone = _emit(rg, [d], prec, 0)
        assert alone[0][1]["chains"] > 100
        _same(alone, [m])
