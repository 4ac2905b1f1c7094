"""Whole steps after a lone emission (rd_do_emission): the emission of the next step feels
the electrons that the lone one added, in either precision.  A field evaluation between the
two brings the FP32 packs up to date by itself, so it must change nothing; and in FP64 the
chains are those of the pair-sum jumps, which read the FP64 positions."""
import numpy as np
import pytest

from test_gpu_near import NM, _electrons, _kw, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("how", ["run", "step", "profile", "serve"])
@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
def test_step_after_lone_emission(rg, prec, how):
    kw = _kw(400.0, 400.0, 6000)
    pos = _electrons(500, 400.0, 400.0, 1000.0, 3)
    res = []
    for kind in ("plain", "field", "atom"):
        with rg.Engine(precision=getattr(rg, prec), max_diodes=2, particle_capacity=6300, chain_capacity=6300,
                       quad_capacity=2 * rg.supply_points(**kw) + 64) as eng:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            if kind == "atom":
                d.add_particle((0.0, 0.0, 500.0 * NM), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            if how == "serve":   # a request that keeps the server running; the diode steps beside it
                eng.submit(5, **dict(_kw(100.0, 100.0, 64), emission=False))
                eng.serve(1)
            eng.do_emission(2)
            if kind == "field":
                d.calc_field_at_batch(np.zeros((1, 3)))
            if how == "run":
                eng.run(3, 2)
            elif how == "step":
                eng.run(3, 1)
                eng.run(4, 1)
            elif how == "profile":
                eng.profile_step(3)
            else:
                eng.serve(2)
            res.append((d.particles(), d.counters()))
    assert res[0][1]["emitted_total"] > 0
    _same(res[:1], res[1:2])
    if prec == "PREC_FP64":
        _same(res[:1], res[2:])
