"""A tip electron that is marked for removal and not yet removed has charge 0, which the
near / far split of the tip's field (rd_tipnear.cuh) does not know: the steps until the
removal take the pair-sum jumps, as launches of their own, instead of sending every jump of
the split through a block's pair sum; the split comes back after it.  Chains, electrons and
counters are those of the pair-sum jumps."""
import numpy as np
import pytest

import test_gpu_tip_near as tip

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("how", ["run", "run3", "remove", "phases", "load"])
def test_marked_electron(rg, how):
    kw, pos = tip._case("close")
    res = []
    for atom in (False, True):
        with rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=15000, chain_capacity=15000,
                       quad_capacity=10064) as eng:
            d = eng.add_diode(geometry=rg.GEOM_TIP, **kw)
            d.add_particles(pos, step=0)
            kernels = []

            def run(k, steps=1):
                eng.run(k, steps)
                kernels.append(eng.last_run_stats()[1])

            if atom:
                d.add_particle((0.0, 0.0, kw["tip_dim"][2] + 0.5 * kw["tip_dim"][0]), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            d.mark_particles_remove(7, rg.REMOVE_TOP)
            if how == "run":
                run(1); run(2)
                want = [True, False]
            elif how == "run3":
                run(1, 3)
                want = [False]
            elif how == "remove":
                eng.remove_particles(0)
                run(1)
                want = [False]
            elif how == "phases":   # one step phase by phase, then a whole one
                eng.do_emission(1)
                eng.update_position(1)
                eng.remove_particles(1)
                run(2)
                want = [False]
            else:
                state = d.save_state()
                eng.remove_particles(0)
                d.load_state(state)
                run(1); run(2)
                want = [True, False]
            res.append((d.particles(), d.counters(), kernels))
    (p, c, kf), (q, s, ks) = res
    assert c["chains"] > 0
    tip._same([(p, c)], [(q, s)])
    assert [k > 80 for k in kf] == want   # 40 jumps of two launches each, or none
