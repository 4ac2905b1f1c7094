"""The jumps of a lone diode start beside other work on the GPU.  Their blocks wait for one
another, so all of them have to be resident at once (a cooperative launch); there are no
more of them than the diode's chains need, and a kernel of another stream that holds a part
of one SM (it spins for about half a second) does not keep a step waiting."""
import pytest

import test_gpu_tip_near as tip
from test_gpu_near import _electrons, _kw

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def busy():
    """An event behind a kernel that runs for about half a second on a stream of its own."""
    s, ev = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(1_000_000_000)
        ev.record(s)
    return ev


@pytest.mark.parametrize("kind", ["fp32", "fp64", "tip"])
def test_step_beside_other_work(rg, kind):
    if kind == "tip":
        kw, pos = tip._case("tile-edge")
        kw = dict(kw, geometry=rg.GEOM_TIP)
    else:
        kw, pos = _kw(300.0, 300.0, 5000), _electrons(400, 300.0, 300.0, 1000.0, 3)
    kw["max_chains"] = 2000
    cap = kw["capacity"] + 64
    with rg.Engine(precision=rg.PREC_FP64 if kind == "fp64" else rg.PREC_FP32C, max_diodes=1, particle_capacity=cap,
                   chain_capacity=cap, quad_capacity=rg.supply_points(**kw) + 64) as eng:
        d = eng.add_diode(**kw)
        d.add_particles(pos, step=0)
        eng.run(1, 1)   # the graph and the kernels are there
        assert d.counters()["chains"] > 0
        torch.cuda.synchronize()
        ev = busy()
        eng.run(2, 2)
        assert not ev.query()   # the other stream's kernel is still running
        torch.cuda.synchronize()
