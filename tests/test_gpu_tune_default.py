"""The default chunking (shorter chunks for small systems) stays in reach: 1024 and 32 stand
for it wherever they come from, so that what get_chunking gives can be set again, the
tuner times it under that name, and a tuned engine's field evaluations, which the tuner
does not time, keep it.  Results are compared bit for bit, which different chunkings of
FP64 partial sums are not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def _diode(rg, n, **cfg):
    r = np.random.default_rng(n)
    p = np.column_stack([r.uniform(-300, 300, n), r.uniform(-300, 300, n), r.uniform(1, 499, n)]) * NM
    eng = rg.Engine(precision=rg.PREC_FP64, max_diodes=1, particle_capacity=n + 64, **cfg)
    d = eng.add_diode(V_s=2.0e3, gap=500 * NM, capacity=n, image_charge=True)
    d.add_particles(p)
    return eng, d, p[:200] * np.array([1.0, 1.0, 0.0])


def _results(d, pts):
    return d.calculate_acceleration_particles(), d.calc_field_at_batch(pts)


@pytest.mark.parametrize("n", [300, 5000])
def test_setting_what_is_set_changes_nothing(rg, n):
    eng, d, pts = _diode(rg, n)
    a, f = _results(d, pts)
    eng.set_chunking(*eng.get_chunking())
    b, g = _results(d, pts)
    eng.close()
    assert np.array_equal(a, b) and np.array_equal(f, g)


@pytest.mark.parametrize("n", [300, 5000])
def test_1024_and_32_are_the_default(rg, n):
    res = []
    for cfg in ({}, dict(chunk_min=1024, chunk_count_max=32)):
        eng, d, pts = _diode(rg, n, **cfg)
        res.append(_results(d, pts))
        eng.set_chunking(512, 8)
        eng.set_chunking(1024, 32)
        res.append(_results(d, pts))
        eng.close()
    for a, f in res[1:]:
        assert np.array_equal(a, res[0][0]) and np.array_equal(f, res[0][1])


def test_tuned_engine_keeps_the_field_rule(rg):
    eng, d, pts = _diode(rg, 9001)
    f = d.calc_field_at_batch(pts)
    t = eng.autotune()
    g = d.calc_field_at_batch(pts)
    eng.set_chunking(2048, 8)
    h = d.calc_field_at_batch(pts)   # by hand: a sum of fewer chunks
    eng.close()
    assert t["ms_chosen"] <= t["ms_default"]
    assert np.array_equal(f, g) and not np.array_equal(f, h)
