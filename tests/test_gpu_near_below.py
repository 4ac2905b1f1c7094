"""Electrons that a caller put below the cathode, or (the tip) inside the apex sphere.  The
bounds of the near / far split (rd_near.cuh, rd_tipnear.cuh) take every term of a sum to
have one sign and every image to lie inside the sphere, so such a diode's next emission
takes the pair-sum jumps -- recognised by the launches of its step -- and the step after
it, when the position update has removed those electrons, the split again.  The chains are
those of the pair-sum jumps either way."""
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


def _below():
    r = np.random.default_rng(11)
    pos = _electrons(1500, 300.0, 300.0, 1000.0, 12)
    low = np.column_stack([r.uniform(-150, 150, 400), r.uniform(-150, 150, 400), r.uniform(-40.0, -0.5, 400)]) * NM
    return dict(_kw(300.0, 300.0, 8000, V=4.0e3, max_chains=3000), mh_jumps=40), np.vstack([pos, low]), {}


def _inside():
    kw, pos = tip._case("close")
    d, R, h = kw["tip_dim"]
    a = np.sqrt((d * d * R * R) / (h * h + 2.0 * d * h) + d * d)
    theta = np.arccos(d / a)
    rad = a * np.sin(theta) * np.tan(theta)
    r = np.random.default_rng(13)
    u = r.normal(size=(50, 3))
    low = np.array([0.0, 0.0, h - rad]) + 0.4 * rad * u / np.linalg.norm(u, axis=1)[:, None]
    return kw, np.vstack([pos, low]), {"geometry": True}


@pytest.mark.parametrize("make,fp64", [(_below, False), (_below, True), (_inside, False)])
@pytest.mark.parametrize("how", ["add", "set", "load", "serve"])
def test_misplaced_electrons(rg, make, fp64, how):
    kw, pos, geo = make()
    if geo:
        kw = dict(kw, geometry=rg.GEOM_TIP)
    cap = kw["capacity"] + 64
    size = dict(precision=rg.PREC_FP64 if fp64 else rg.PREC_FP32C, particle_capacity=cap,
                chain_capacity=cap + kw.get("max_chains", 0), quad_capacity=rg.supply_points(**kw) + 64, max_diodes=1)
    res = []
    for atom in (False, True):
        with rg.Engine(**size) as eng:
            kernels = []
            if how == "serve" and not atom:
                rid = eng.submit(1000, pos=pos, **kw)
                for _ in range(2):
                    eng.serve(1)
                    kernels.append(eng.last_run_stats()[1])
                d = rg.Diode(eng, 0)
            else:
                d = eng.add_diode(**kw)
                if atom:
                    d.add_particle((0.0, 0.0, 900.0 * NM), species=rg.ATOM, step=0)
                    d.mark_particles_remove(0, rg.REMOVE_TOP)
                    eng.remove_particles(0)
                if how == "set":   # placed well first, then moved
                    d.add_particles(np.repeat([[0.0, 0.0, 900.0 * NM]], len(pos), axis=0), step=0)
                    d.set_particles(pos=pos)
                else:
                    d.add_particles(pos, step=0)
                if how == "load" and not atom:
                    state = d.save_state()
                    eng.remove_diode(d)
                    d = eng.add_diode(**kw)
                    d.load_state(state)
                for k in (1, 2):
                    eng.run(k, 1)
                    kernels.append(eng.last_run_stats()[1])
            res.append((d.particles(), d.counters(), kernels))
    (p, c, kf), (q, s, ks) = res
    assert c["chains"] > 0
    _same([(p, c)], [(q, s)])
    # 40 jumps with launches of their own, or none
    assert [k > 55 for k in kf] == [True, False] and [k > 55 for k in ks] == [True, True]
