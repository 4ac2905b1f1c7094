"""The near / far split of the chains' field (rd_near.cuh) against the pair-sum
jumps.  A diode that was given an atom keeps the pair-sum kernel, also after the atom
has left, so the same diode with and without that history has to run the same
chains: every electron, counter and step size equal, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM = 1.0e-9
COUNTS = ("n", "emitted_total", "dropped_total", "absorbed_top_total", "absorbed_bot_total", "chains", "chains_failed")


@pytest.fixture(scope="module")
def rg():
    import rumdeed_gb300
    rumdeed_gb300.build()
    return rumdeed_gb300


def _kw(side_x, side_y, cap, V=2.0e3, gap=1000.0, work=((2.0,),), **more):
    return dict(V_s=V, gap=gap * NM, time_step=0.25e-15, image_charge=True, N_ic_max=0, capacity=cap,
                emitter_pos=(-side_x / 2 * NM, -side_y / 2 * NM), emitter_dim=(side_x * NM, side_y * NM),
                work=[list(r) for r in work], emission=True, seed=77, mh_jumps=40, **more)


def _electrons(n, side_x, side_y, gap, seed, low=3):
    """n electrons, most of them close to the cathode, some outside the emitter's footprint."""
    r = np.random.default_rng(seed)
    z = 1.0 + (gap - 2.0) * r.uniform(0.0, 1.0, n) ** low
    return np.column_stack([r.uniform(-0.6, 0.6, n) * side_x, r.uniform(-0.6, 0.6, n) * side_y, z]) * NM


def _run(rg, diodes, steps, atom, chunk=None, fp64=False):
    quad = sum(rg.supply_points(**kw) for kw, _ in diodes) + 64 * len(diodes)
    cap = sum(kw["capacity"] + 64 for kw, _ in diodes)
    chains = sum(max(kw["capacity"], kw.get("max_chains", 0)) + 64 for kw, _ in diodes)
    with rg.Engine(precision=rg.PREC_FP64 if fp64 else rg.PREC_FP32C, max_diodes=len(diodes), particle_capacity=cap, chain_capacity=chains,
                   quad_capacity=quad) as eng:
        if chunk:
            eng.set_chunking(*chunk)
        out = []
        for kw, pos in diodes:
            d = eng.add_diode(**kw)
            if len(pos):
                d.add_particles(pos, step=0)
            if atom:
                d.add_particle((0.0, 0.0, 0.5 * kw["gap"]), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            out.append(d)
        eng.run(1, steps)
        assert sum(eng.validate().values()) == 0
        res = []
        for d in out:
            res.append((d.particles(), d.counters()))
        return res


def _same(a, b):
    for (p, c), (q, e) in zip(a, b):
        for k in ("pos", "vel", "acc", "charge", "section"):
            assert np.array_equal(p[k], q[k]), k
        for k in COUNTS:
            assert c[k] == e[k], k
        for k in ("N_sup", "MH_std", "a_rate", "residual", "df_avg", "F_avg", "ramo_current"):
            assert c[k] == e[k], k


CHECKER = ((2.0, 2.6), (2.3, 1.9))
CASES = {
    # electrons, emitter (nm), gap, options
    "no-low-electrons": (129, 500.0, 500.0, 1000.0, dict(low=0.1)),
    "few": (33, 1000.0, 1000.0, 1000.0, {}),
    "tile-edge": (128, 310.0, 330.0, 400.0, {}),
    "small-emitter": (2001, 100.0, 100.0, 300.0, {}),
    "oblong": (3000, 700.0, 400.0, 800.0, dict(work=CHECKER)),
    "layers": (5000, 1000.0, 1000.0, 1000.0, {}),
    "many-chains": (4000, 2000.0, 1900.0, 1000.0, dict(V=2.2e3, max_chains=20000)),
}


CHUNKED = [(name, chunk) for name in ("layers", "tile-edge") for chunk in ((128, 32), (2048, 4))]


@pytest.mark.parametrize("name,chunk", [(name, None) for name in sorted(CASES)] + CHUNKED)
def test_near_far_chains_equal_pair_sum_chains(rg, name, chunk):
    n, lx, ly, gap, opt = CASES[name]
    opt = dict(opt)
    pos = _electrons(n, lx, ly, gap, 5, opt.pop("low", 3))
    kw = _kw(lx, ly, n + 6000, gap=gap, **opt)
    fast, slow = (_run(rg, [(kw, pos)], 3, atom, chunk) for atom in (False, True))
    assert fast[0][1]["emitted_total"] > 0
    _same(fast, slow)


@pytest.mark.parametrize("name,chunk", [(name, None) for name in sorted(CASES)] + [("tile-edge", (128, 32))])
def test_near_far_fp64_chains_equal_pair_sum_chains(rg, name, chunk):
    n, lx, ly, gap, opt = CASES[name]
    opt = dict(opt)
    pos = _electrons(n, lx, ly, gap, 6, opt.pop("low", 3))
    kw = _kw(lx, ly, n + 6000, gap=gap, **opt)
    fast, slow = (_run(rg, [(kw, pos)], 3, atom, chunk, fp64=True) for atom in (False, True))
    assert fast[0][1]["emitted_total"] > 0
    _same(fast, slow)


def test_near_far_fp64_mix_equals_alone(rg):
    sizes = [(700, 200.0, 300.0), (900, 900.0, 700.0), (60, 1500.0, 1000.0)]
    diodes = [(dict(_kw(s, s, n + 3000, gap=g), seed=100 + k), _electrons(n, s, s, g, k))
              for k, (n, s, g) in enumerate(sizes)]
    mix = _run(rg, diodes, 3, False, fp64=True)
    for k, d in enumerate(diodes):
        _same(_run(rg, [d], 3, False, fp64=True), mix[k:k + 1])


def test_emission_after_emission(rg):
    """Two emissions without a position update between them: the second one's
    chains feel the first one's electrons."""
    kw = _kw(400.0, 400.0, 4000)
    pos = _electrons(500, 400.0, 400.0, 1000.0, 3)
    res = []
    for atom in (False, True):
        with rg.Engine(precision=rg.PREC_FP64, max_diodes=1, particle_capacity=4100, chain_capacity=4100,
                       quad_capacity=rg.supply_points(**kw) + 64) as eng:
            d = eng.add_diode(**kw)
            d.add_particles(pos, step=0)
            if atom:
                d.add_particle((0.0, 0.0, 500.0 * NM), species=rg.ATOM, step=0)
                d.mark_particles_remove(len(pos), rg.REMOVE_TOP)
                eng.remove_particles(0)
            eng.do_emission(1)
            eng.do_emission(2)
            res.append((d.particles(), d.counters()))
    assert res[0][1]["emitted_total"] > 0
    _same(res[:1], res[1:])


def test_near_far_mix_equals_alone(rg):
    sizes = [(700, 200.0, 300.0), (2500, 900.0, 700.0), (60, 1500.0, 1000.0), (4100, 600.0, 500.0)]
    diodes = [(dict(_kw(s, s, n + 3000, gap=g), seed=100 + k), _electrons(n, s, s, g, k))
              for k, (n, s, g) in enumerate(sizes)]
    mix = _run(rg, diodes, 3, False)
    for k, d in enumerate(diodes):
        _same(_run(rg, [d], 3, False), mix[k:k + 1])


def test_loaded_atom_keeps_the_pair_sum(rg):
    """A checkpoint that holds an atom, loaded into a diode that had none."""
    kw = _kw(400.0, 400.0, 4000)
    pos = _electrons(900, 400.0, 400.0, 1000.0, 9)

    def engine():
        return rg.Engine(precision=rg.PREC_FP32C, max_diodes=1, particle_capacity=4100, chain_capacity=4100,
                         quad_capacity=rg.supply_points(**kw) + 64)

    with engine() as a, engine() as b:
        d = a.add_diode(**kw)
        d.add_particles(pos, step=0)
        d.add_particle((0.0, 0.0, 500.0 * NM), species=rg.ATOM, step=0)
        a.run(1, 1)
        state = d.save_state()
        e = b.add_diode(**kw)
        b.run(1, 1)
        e.load_state(state)
        a.run(2, 2)
        b.run(2, 2)
        _same([(d.particles(), d.counters())], [(e.particles(), e.counters())])
