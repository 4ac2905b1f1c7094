"""Particles and points through the pinned transfer buffer (k_rows_out, k_points_in /
_out, k_state_in): whatever goes in comes back, for the smallest and odd counts, for
more rows than one part of the buffer holds, with a caller's arrays shorter than the
diode, and for accelerations asked for right after an emission, whose electrons no
position update has packed yet."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def _state(n, seed=1):
    r = np.random.default_rng(seed)
    p = np.column_stack([r.uniform(-500, 500, n), r.uniform(-500, 500, n), r.uniform(1, 999, n)]) * NM
    return p, r.normal(0.0, 1.0e5, (n, 3))


@pytest.mark.parametrize("n", [0, 1, 85, 86, 257, 100003, 1000001])   # the last: two parts
def test_particles_come_back(rg, n):
    pos, vel = _state(n)
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=2, particle_capacity=2 * n + 200) as eng:
        d = eng.add_diode(V_s=2.0e3, gap=1000 * NM, capacity=n + 64)
        if n:
            d.add_particles(pos, vel, step=0)
        p = d.particles()
        assert d.n == n and len(p["id"]) == n
        np.testing.assert_array_equal(p["pos"], pos)
        np.testing.assert_array_equal(p["vel"], vel)
        np.testing.assert_array_equal(p["id"], np.arange(n))
        e = eng.add_diode(V_s=2.0e3, gap=1000 * NM, capacity=n + 64)
        e.load_state(d.save_state())
        q = e.particles()
        for k in p:
            np.testing.assert_array_equal(p[k], q[k], err_msg=k)
        few = np.full((7, 3), -1.0)
        nout = C.c_int()
        rg._check(eng.L.rd_get_particles(eng.h, d.index, 5, few.ctypes.data_as(C.POINTER(C.c_double)), None, None, None,
                                         None, None, C.byref(nout)))
        m = min(n, 5)
        assert nout.value == n and np.all(few[m:] == -1.0)
        np.testing.assert_array_equal(few[:m], pos[:m])


@pytest.mark.parametrize("m", [1, 127, 129, 5000])
def test_fields_come_back_in_order(rg, m):
    pos, _ = _state(300)
    pts, _ = _state(m, 2)
    with rg.Engine(precision=rg.PREC_FP64, max_diodes=3, particle_capacity=2000) as eng:
        ds = [eng.add_diode(V_s=2.0e3, gap=1000 * NM, capacity=400) for _ in range(3)]
        for d in ds:
            d.add_particles(pos)
        all_ = ds[1].calc_field_at_batch(pts)
        one = np.vstack([ds[2].calc_field_at_batch(pts[k:k + 1]) for k in (0, m // 2, m - 1)])
        np.testing.assert_array_equal(all_[[0, m // 2, m - 1]], one)


def test_forces_after_an_emission_see_its_electrons(rg):
    kw = dict(V_s=2.0e3, gap=1000 * NM, capacity=4000, emitter_pos=(-200 * NM, -200 * NM),
              emitter_dim=(400 * NM, 400 * NM), work=[[2.0]], emission=True, mh_jumps=20, seed=5)
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=4100, chain_capacity=4100) as eng:
        d = eng.add_diode(**kw)
        eng.do_emission(1)
        assert d.n > 20
        a = d.calculate_acceleration_particles()
        p = d.particles()["pos"]
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=4100, chain_capacity=4100) as eng:
        d = eng.add_diode(**kw)
        d.add_particles(p)
        np.testing.assert_array_equal(a, d.calculate_acceleration_particles())
