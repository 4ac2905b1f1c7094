"""The default j-chunking shortens the chunks of small systems (k_plan) so that they
fill the GPU.  Chunk partials are added in FP64 (or as float pairs of ~44 bits), so the
results agree with any fixed chunking far below the FP32 form's tolerance, a chunking
set by hand is kept, and 0, 0 brings the default back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("n", [1, 127, 129, 1024, 1025, 5000, 40000])
@pytest.mark.parametrize("prec", ["PREC_FP32C", "PREC_FP64"])
def test_default_chunking_equals_fixed_ones(rg, n, prec):
    if prec == "PREC_FP64" and n > 5000:
        n = 9001
    r = np.random.default_rng(n)
    p = np.column_stack([r.uniform(-300, 300, n), r.uniform(-300, 300, n), r.uniform(1, 499, n)]) * NM
    pts = p[: min(n, 300)] * np.array([1.0, 1.0, 0.0])
    got = []
    with rg.Engine(precision=getattr(rg, prec), max_diodes=1, particle_capacity=n + 64) as eng:
        d = eng.add_diode(V_s=2.0e3, gap=500 * NM, capacity=n, image_charge=True)
        d.add_particles(p)
        for chunk in (None, (1024, 32), (65408, 1), (0, 0)):
            if chunk:
                eng.set_chunking(*chunk)
            assert eng.get_chunking() == (chunk if chunk and chunk[0] else (1024, 32))
            got.append((d.calculate_acceleration_particles(), d.calc_field_at_batch(pts)))
    for a, f in got[1:]:
        assert np.max(np.abs(a - got[0][0])) <= 1e-12 * np.max(np.abs(a))
        assert np.max(np.abs(f - got[0][1])) <= 1e-12 * np.max(np.abs(f))
    np.testing.assert_array_equal(got[0][0], got[3][0])
    np.testing.assert_array_equal(got[0][1], got[3][1])
