"""The serial sampler's decisions from float fields (k_mh_serial, FP32 form): chain for
chain the oracle's FP64 sampler.  The field of the FP32 form is within 1e-6 of the
oracle's, a decision closer than that to its threshold has a chance of about 1e-6, and
a case makes at most 6000 jumps, so every electron, count and step size agrees.  Jump
counts around the 256 draws a block holds, particle counts around a warp, the block
and its four loads in flight, and the work-function models with and without cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.fixture(scope="module")
def orc():
    import os
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
    import orc
    orc.build()
    return orc


CHECKER = [[2.0, 2.4], [2.2, 1.9]]
CASES = [(1, 40, [[2.0]]), (31, 256, [[2.0]]), (33, 257, CHECKER), (255, 300, [[2.0]]), (257, 40, CHECKER),
         (1024, 40, [[2.0]]), (1025, 41, CHECKER)]


@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
@pytest.mark.parametrize("n0,jumps,work", CASES)
def test_serial_chains_match_oracle(rg, orc, prec, n0, jumps, work):
    r = np.random.default_rng(n0)
    d, V = 500 * NM, 1.0e3
    pos = np.column_stack([r.uniform(-60, 60, n0), r.uniform(-60, 60, n0), r.uniform(2, 490, n0)]) * NM
    o = orc.OracleDiode(cap=4096, V_s=V, d=d)
    o.set_planar_emitter(-50 * NM, -50 * NM, 100 * NM, 100 * NM, work)
    o.set_emission(True, seed=31, mh_jumps=jumps, max_chains=20, quad_panels=8, quad_order=4)
    o.s.mh_serial = 1
    o.add_many(pos)
    o.emission(1)
    with rg.Engine(precision=getattr(rg, prec), max_diodes=1, particle_capacity=8192, chain_capacity=4096) as eng:
        dio = eng.add_diode(V_s=V, gap=d, capacity=4096, emitter_pos=(-50 * NM, -50 * NM),
                            emitter_dim=(100 * NM, 100 * NM), work=work, emission=True, mh_jumps=jumps, max_chains=20,
                            quad_panels=8, quad_order=4, seed=31, mh_serial=True)
        dio.add_particles(pos)
        eng.do_emission(1)
        c, p = dio.counters(), dio.particles()
    assert c["chains"] == 20 and c["emitted_step"] == o.s.emitted_step
    assert c["MH_std"] == pytest.approx(o.s.MH_std, rel=1e-12)
    assert c["df_avg"] == pytest.approx(o.s.df_avg, rel=1e-4 if prec == "PREC_FP32C" else 1e-10)
    assert dio_equal(p["pos"], o.arr("pos")[:o.n])


def dio_equal(a, b):
    return len(a) == len(b) and (len(a) == 0 or np.max(np.abs(a - b)) < 1e-12 * 100 * NM)
