"""The near / far split of the FP32 tip chains' field (rd_tipnear.cuh) against the
pair-sum jumps.  A diode that was given an atom keeps the pair-sum kernel, also after the
atom has left, so the same diode with and without that history has to run the same
chains: every electron, counter and step size equal, bit for bit."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def _tip(apex, gap, high=500.0):
    """(d_tip, R_base, h_tip) of a hyperboloid with this apex radius (nm)."""
    h, d = high * NM, gap * NM
    return d, math.sqrt(apex * NM * ((h * h) / d + 2.0 * h)), h


def _cloud(dims, n, seed, low):
    """n electrons in front of the tip, more of them close to it for a larger `low`."""
    d, R, h = dims
    a = math.sqrt((d * d * R * R) / (h * h + 2.0 * d * h) + d * d)
    eta1, ximax = -d / a, h / d + 1.0
    r = np.random.default_rng(seed)
    xi = 1.0 + 0.9 * (ximax - 1.0) * r.uniform(0.0, 1.0, n)
    eta = eta1 * (1.0 - 0.9 * (0.002 + r.uniform(0.0, 1.0, n) ** low))
    phi = r.uniform(0.0, 2.0 * np.pi, n)
    xy = a * np.sqrt((xi * xi - 1.0) * (1.0 - eta * eta))
    return np.column_stack([xy * np.cos(phi), xy * np.sin(phi), a * xi * eta + abs(a * eta1 * ximax)])


def _kw(dims, cap, V, **more):
    return dict(dict(V_s=V, time_step=0.25e-15, image_charge=True, N_ic_max=0, capacity=cap, tip_dim=dims,
                     emission=True, seed=77, mh_jumps=40), **more)


def _run(rg, diodes, steps, atom, chunk=None):
    quad = 10064 * len(diodes)
    cap = sum(kw["capacity"] + 64 for kw, _ in diodes)
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=len(diodes), particle_capacity=cap, chain_capacity=cap,
                   quad_capacity=quad) as eng:
        if chunk:
            eng.set_chunking(*chunk)
        out = []
        for k, (kw, pos) in enumerate(diodes):
            d = eng.add_diode(geometry=rg.GEOM_TIP, **kw)
            if len(pos):
                d.add_particles(pos, step=0)
            if atom is True or (atom and atom[k]):
                d.add_particle((0.0, 0.0, kw["tip_dim"][2] + 0.5 * kw["tip_dim"][0]), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            out.append(d)
        eng.run(1, steps)
        assert sum(eng.validate().values()) == 0
        return [(d.particles(), d.counters()) for d in out]


def _same(a, b):
    for (p, c), (q, e) in zip(a, b):
        for k in ("pos", "vel", "acc", "charge", "section"):
            assert np.array_equal(p[k], q[k]), k
        for k in ("n", "emitted_total", "dropped_total", "absorbed_top_total", "absorbed_bot_total", "chains",
                  "chains_failed", "N_sup", "MH_std", "a_rate", "residual", "df_avg", "ramo_current"):
            assert c[k] == e[k], k


CASES = {
    # electrons, apex radius (nm), gap, how close to the tip, options
    "none": (0, 100.0, 1000.0, 1, dict(V=1500.0)),
    "one": (1, 100.0, 1000.0, 4, dict(V=1500.0)),
    "tile-edge": (128, 250.0, 1000.0, 3, dict(V=2000.0)),
    "sharp": (2001, 20.0, 500.0, 3, dict(V=800.0)),
    "blunt": (3000, 400.0, 300.0, 3, dict(V=1500.0)),
    "close": (5000, 250.0, 1000.0, 6, dict(V=3000.0)),
    "spread": (9000, 250.0, 1000.0, 1, dict(V=2500.0)),
    "no-image": (2000, 150.0, 1000.0, 3, dict(V=2000.0, image_charge=False)),
    "work": (1500, 250.0, 1000.0, 3, dict(V=1500.0, tip_work_function=3.0)),
}


def _case(name):
    n, apex, gap, low, opt = CASES[name]
    dims = _tip(apex, gap)
    return _kw(dims, n + 9000, **opt), _cloud(dims, n, 5, low)


@pytest.mark.parametrize("name,chunk", [(name, None) for name in sorted(CASES)] +
                         [("close", (128, 32)), ("close", (2048, 4)), ("tile-edge", (128, 32))])
def test_near_far_tip_chains_equal_pair_sum_chains(rg, name, chunk):
    d = _case(name)
    fast, slow = (_run(rg, [d], 3, atom, chunk) for atom in (False, True))
    assert fast[0][1]["chains"] > 0
    _same(fast, slow)


def test_tip_mix_equals_alone(rg):
    """Tips of both kinds of jumps side by side, with different numbers of jumps."""
    diodes = [_case("sharp"), _case("close"), _case("tile-edge"), _case("work")]
    diodes = [(dict(kw, seed=100 + k, mh_jumps=20 + 10 * k), pos) for k, (kw, pos) in enumerate(diodes)]
    mix = _run(rg, diodes, 3, (False, True, True, False))
    for k, d in enumerate(diodes):
        _same(_run(rg, [d], 3, False), mix[k:k + 1])


def test_list_memory_follows_the_diodes(rg):
    """Adding and removing tips gives their lists back."""
    import torch
    kw, pos = _case("close")
    with rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=15000, chain_capacity=15000,
                   quad_capacity=10064) as eng:
        free = []
        for _ in range(3):
            d = eng.add_diode(geometry=rg.GEOM_TIP, **kw)
            d.add_particles(pos, step=0)
            eng.run(1, 1)
            eng.remove_diode(d)
            free.append(torch.cuda.mem_get_info()[0])
        assert free[1] == free[2]
