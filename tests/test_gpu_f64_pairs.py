"""The FP64 pair sums' inverse cubes (rd_f64.cuh) over the whole range of distances,
against the oracle's sqrt and division: pairs just below and above the 2 nm where the
series takes over from the plain formula, coincident electrons, a millimetre apart,
planar and tip, as forces and as fields.  Each term carries at most 2.3 u (u = 1.1e-16)
against the oracle's 5.7 u, and a few hundred are added, so 1e-12, the FP64 form's
tolerance, leaves room for the cancellation of a few decades."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9
TOL = 1.0e-12


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


def _nrel(a, b):
    return np.max(np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1))


def _cluster(n, seed, centre, far):
    """n points: steps of 1e-3 .. 4 nm from one to the next, some exactly at and around 2 nm."""
    r = np.random.default_rng(seed)
    u = r.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    step = np.where(np.arange(n) % 3 == 0, 2.0 + r.uniform(-1e-6, 1e-6, n), 10.0 ** r.uniform(-3, np.log10(4.0), n))
    p = np.cumsum(u * step[:, None], axis=0)
    p += np.asarray(centre) - p.mean(axis=0)
    p[:, 2] = np.abs(p[:, 2]) + 0.5
    if n > 3:
        p[n // 2] += far
    return p * NM


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 300])
@pytest.mark.parametrize("nic", [0, 2])
def test_planar_pairs_match_oracle(rg, orc, n, nic):
    p = _cluster(n, n, (0.0, 0.0, 40.0), (1.0e6, 0.0, 0.0))   # one electron 1 mm away
    if n > 100:
        p[-1] = p[0]   # coincident: the pair's force is 0
    o = orc.OracleDiode(cap=1024, V_s=2.0e3, d=1000 * NM, image_charge=True, N_ic_max=nic)
    o.add_many(p)
    pts = np.vstack([p[:20] + np.array([0.0, 0.0, 0.3]) * NM, [[0.0, 0.0, 0.0], [2.0e-3, 0.0, 500.0 * NM]]])
    with rg.Engine(precision=rg.PREC_FP64, max_diodes=1, particle_capacity=4096) as eng:
        d = eng.add_diode(V_s=2.0e3, gap=1000 * NM, capacity=1024, image_charge=True, N_ic_max=nic)
        d.add_particles(p)
        assert _nrel(d.calculate_acceleration_particles(), o.accel("gather", True)) <= TOL
        assert _nrel(d.calc_field_at_batch(pts), o.field_at(pts)) <= TOL


@pytest.mark.parametrize("n", [1, 2, 128, 129, 300])
@pytest.mark.parametrize("ic", [True, False])
def test_tip_pairs_match_oracle(rg, orc, n, ic):
    tip = (900 * NM, 100 * NM, 100 * NM)
    p = _cluster(n, 7 * n, (20.0, 10.0, 160.0), (0.0, 0.0, 500.0))
    o = orc.OracleDiode(orc.TIP, cap=1024, V_s=2.0e3, d=1000 * NM, image_charge=ic)
    o.set_tip(*tip, 4.7)
    o.add_many(p)
    pts = p[:20] + np.array([0.4, 0.0, 0.0]) * NM
    with rg.Engine(precision=rg.PREC_FP64, max_diodes=1, particle_capacity=4096) as eng:
        d = eng.add_diode(geometry=rg.GEOM_TIP, V_s=2.0e3, capacity=1024, tip_dim=tip, image_charge=ic)
        d.add_particles(p)
        assert _nrel(d.calculate_acceleration_particles(), o.accel("gather", True)) <= TOL
        assert _nrel(d.calc_field_at_batch(pts), o.field_at(pts)) <= TOL
