"""The FP32 field at points of a planar diode with one image partner or none
(k_field_points: two points per thread, half of a tile each; more chunks per tile)
against the FP64 form.  A term is good to 25 u (u = 2^-24: differences, reciprocal
root, products) and a run of at most 64 terms adds at most 64 u of the sum of
magnitudes; positions agree to 2^-45 of the emitter's size.  The tolerance is 100 u
of the terms' magnitudes at each point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


@pytest.mark.parametrize("image", [True, False])
@pytest.mark.parametrize("n,m", [(0, 5), (1, 1), (2, 64), (64, 65), (127, 63), (128, 128), (129, 129), (1000, 1),
                                 (1025, 130), (12500, 257)])
@pytest.mark.parametrize("ions", [False, True])
def test_planar_field_points(rg, n, m, image, ions):
    r = np.random.default_rng(1000 * n + m)
    gap = 600.0
    p = np.column_stack([r.uniform(-300, 300, n), r.uniform(-300, 300, n), r.uniform(1, gap - 1, n)])
    q = np.column_stack([r.uniform(-300, 300, m), r.uniform(-300, 300, m), r.uniform(0, gap, m)])
    q[::3, 2] = 0.0
    species = np.where(r.uniform(size=n) < 0.3, rg.ION, rg.ELEC) if ions else None
    f = []
    for prec in (rg.PREC_FP32C, rg.PREC_FP64):
        with rg.Engine(precision=prec, max_diodes=1, particle_capacity=n + 64) as eng:
            d = eng.add_diode(V_s=2.0e3, gap=gap * NM, capacity=n + 16, image_charge=image, N_ic_max=0)
            if n:
                d.add_particles(p * NM, species=species)
            f.append(np.asarray(d.calc_field_at_batch(q * NM)))
    mag = np.zeros(m)
    for k in range(n):
        dx = q - p[k]
        mag += 1.0 / np.maximum((dx * dx).sum(1), 1e-20)
        if image:
            dx = q - p[k] * np.array([1, 1, -1])
            mag += 1.0 / np.maximum((dx * dx).sum(1), 1e-20)
    k = rg.q_0 / (4.0 * np.pi * 8.8541878128e-12) * 1.0e18
    tol = 100.0 * 2.0 ** -24 * k * mag[:, None] + 1.0e-12 * np.abs(f[1])
    assert np.all(np.abs(f[0] - f[1]) <= tol)
