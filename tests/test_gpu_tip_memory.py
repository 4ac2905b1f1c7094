"""The memory of a tip's panels and lists comes and goes in stream order: adding or removing
an emitting FP32 tip, by hand or by the server, waits for no other work on the GPU (a
kernel of another stream that spins for about half a second)."""

import pytest

import test_gpu_tip_near as tip
from test_gpu_beside import busy

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("how", ["add", "serve"])
def test_tips_come_and_go_beside_other_work(rg, how):
    kw, pos = tip._case("tile-edge")
    kw = dict(kw, geometry=rg.GEOM_TIP, max_chains=2000)
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=2, particle_capacity=20000, chain_capacity=20000,
                   quad_capacity=20128) as eng:

        def cycle():
            if how == "add":
                d = eng.add_diode(**kw)
                d.add_particles(pos, step=0)
                eng.run(1, 1)
                eng.remove_diode(d)
            else:
                for _ in range(2):
                    eng.submit(1, pos=pos, **kw)
                while eng.serve(1)["running"]:
                    pass

        cycle()
        torch.cuda.synchronize()
        ev = busy()
        cycle()
        assert not ev.query()   # the other stream's kernel is still running
        torch.cuda.synchronize()
