"""Launch shapes that depend on the size of the work: every shape gives the same bits, and the
smallest one agrees with the FP64 oracle engine."""
import threading

import numpy as np
import pytest

import mdpd
import oracle

pytestmark = pytest.mark.gpu

RHO = 6.05


def lattice(n, L, seed):
    """n sites of a jittered cubic lattice and Maxwell velocities"""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    s = rng.permutation(m ** 3)[:n]
    x = (np.stack([s % m, s // m % m, s // m // m], 1) + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) * (L / m)
    v = rng.normal(0, 1, (n, 3))
    return x, v - v.mean(0)


# the box sizes: a row block cut short (401 = 3 x 128 + 17), whole blocks, one row past a block
@pytest.mark.parametrize("n", [401, 2048, 2049])
@pytest.mark.parametrize("exact", [0, 1])
def test_small_box_same_bits_in_any_mix_and_close_to_the_oracle(n, exact):
    """alone the box takes the shapes of the smallest work; beside boxes of 20k, 100k and 700k
    particles those of the larger ranges"""
    L = (n / RHO) ** (1 / 3)
    x, v = lattice(n, L, 5)
    spec = mdpd.box_spec(n, L, x=x, v=v, seed=77, exact_rng=exact)
    got = []
    for other in (0, 20000, 100000, 700000):
        sp = [spec]
        if other:
            sp.append(mdpd.box_spec(other, (other / RHO) ** (1 / 3), seed=5, init_seed=3, exact_rng=exact))
        b = mdpd.Batch(sp)
        b.setup()
        b.step(5)
        got.append(b.state(0))
        b.step(7)
        got[-1] += b.state(0)
        b.close()
    for g in got[1:]:
        for a, c in zip(got[0], g):
            assert np.array_equal(a, c)
    # 5 steps, each adding to v at most dt times the force bar (1e-5 of the RMS force, ~60) and, with
    # the FP32 gaussian, its error (3e-6) in ~25 random pair forces of sigma w_c / sqrt(dt) ~ 10 each;
    # half as much again for growth
    sim = oracle.Sim(x, v, (0, 0, 0), (L, L, L), seed=77)
    sim.setup()
    sim.run(5)
    xo, vo = sim.state()[:2]
    sim.close()
    bar = 1.5 * 5 * 0.01 * (1e-5 * 60 + 25 * 10 * 3e-6)
    assert np.abs(got[0][1] - vo).max() < bar
    dx = got[0][0] - xo
    assert np.abs(dx - L * np.round(dx / L)).max() < 5 * 0.01 * bar


def test_ghost_overflow_is_reported_and_the_library_stays_usable():
    """every particle within the ghost cutoff of a face: more images than the capacity estimated
    for a uniform box"""
    L = 40.0
    n = int(RHO * 1.2 * L * L)
    rng = np.random.default_rng(2)
    x = rng.uniform(0, 1, (n, 3)) * (1.2, L, L)
    b = mdpd.Batch([mdpd.box_spec(n, L, x=x, v=np.zeros((n, 3)))])
    with pytest.raises(mdpd.MdpdError) as e:
        b.setup()
    assert e.value.code == mdpd.ERR_OVERFLOW and "ghost" in str(e.value)
    b.close()
    m = 2000
    b = mdpd.Batch([mdpd.box_spec(m, (m / RHO) ** (1 / 3))])
    b.setup()
    b.step(3)
    assert b.thermo(0).status == 0
    b.close()


def deck(n, lo, hi, types, pair, fixes, x, v, style="mdpd"):
    lam = mdpd.Lammps()
    lam.commands(f"units lj\nboundary p p p\nneighbor 0.3 bin\nneigh_modify every 1 delay 0 check yes\n"
                 f"atom_style {style}/atomic/meso 8\n"
                 f"region box block {lo[0]} {hi[0]} {lo[1]} {hi[1]} {lo[2]} {hi[2]} units box\n"
                 f"create_box {len(n)} box")
    for t, c in enumerate(n):
        lam.command(f"create_atoms {t + 1} random {c} {11 + t} box")
        lam.command(f"mass {t + 1} 1")
    lam.commands(types)
    lam.commands(pair)
    lam.commands(fixes)
    lam.commands("timestep 0.01\nrun_style mvv/meso")
    lam.set_state(x, v)
    return lam


FIELDS = ("tag", "x", "v", "force")


def fields(lam, names=FIELDS):
    return [lam.field(k) for k in names]


def same(a, b):
    return all(np.array_equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("exact", ["yes", "no"])
def test_steps_of_one_run_same_bits_as_single_runs(exact):
    """12 steps of one call leave each step's final half-kick to the next step; single steps apply
    it themselves.  One group frozen, one under a body force."""
    n, L = 3001, 8.0
    x, v = lattice(n, L, 9)
    mk = lambda: deck((2000, 1001), (0,) * 3, (L,) * 3,  # noqa: E731
                      "group mov type 1\ngroup fix type 2",
                      "pair_style mdpd/meso 1.0 1.0 77\npair_coeff * * -40 25 4.5 1.0 0.75\n"
                      f"pair_modify rng {'exact' if exact == 'yes' else 'fast'}",
                      "fix R all aboundary/rho/meso cut_rho 0.75\nfix N mov nve/meso\nfix F mov addforce/meso 0.02 0.0 -0.01",
                      x, v)
    a, b = mk(), mk()
    a.setup()
    b.setup()
    a.step(12)
    for _ in range(12):
        b.step(1)
    assert same(fields(a), fields(b))
    a.run(2)  # a step with energy and virial after deferred ones
    b.run(2)
    assert same(fields(a), fields(b))
    a.close()
    b.close()


def dpd_box(n, exact):
    L = (n / 3.0) ** (1 / 3)
    x, v = lattice(n, L, 6)
    return deck((n - n // 4, n // 4), (0,) * 3, (L,) * 3, "group all2 type 2",
                "pair_style dpd/meso 1.0 77\npair_coeff 1 1 25 4.5 3.0 1.0 1.0\npair_coeff 1 2 30 4.5 3.0 1.0 0.9\n"
                f"pair_coeff 2 2 20 4.5 3.0 1.0 1.0\npair_modify rng {exact}", "fix NVE all nve/meso", x, v, "dpd")


def mdpd_box(n, exact):
    L = (n / RHO) ** (1 / 3)
    x, v = lattice(n, L, 8)
    return deck((n - n // 4, n // 4), (0,) * 3, (L,) * 3, "group one type 1",
                "pair_style mdpd/meso 1.0 1.0 77\npair_coeff 1 1 -40 25 4.5 1.0 0.75\n"
                "pair_coeff 1 2 -35 25 4.5 0.9 0.7\npair_coeff 2 2 -45 25 4.5 1.0 0.75\n"
                f"pair_modify rng {exact}",
                "fix R all aboundary/rho/meso cut_rho 0.75\nfix N all nve/meso\nfix F one addforce/meso 0.02 0.0 -0.01", x, v)


# one block per SM holds 1/148 of the rows: boxes at the edges of the lanes-per-row ranges (24 and 96
# rows per block on a B200), below and above one row per block, and some way into the range of two lanes
@pytest.mark.parametrize("exact", ["fast", "exact"])
@pytest.mark.parametrize("n", [401, 3552, 3553, 14208, 14209, 30011, 70001])
@pytest.mark.parametrize("make", [mdpd_box, dpd_box])
def test_runs_of_a_small_box_same_bits_as_step_by_step(make, n, exact):
    """without thermo output the steps of a run go in one launch; a thermo line at every step makes
    each a launch of its passes (with energy and virial).  Rebuilds, types, groups, a body force."""
    a, b = make(n, exact), make(n, exact)
    b.command("thermo 1")
    steps = 270 if n < 1000 else 14  # past one launch's 256 steps
    a.run(steps)
    b.run(steps)
    assert a.thermo().nbuild == b.thermo().nbuild >= 3
    assert same(fields(a, FIELDS + ("rho",)), fields(b, FIELDS + ("rho",)))
    assert same(a.list_rows(), b.list_rows())
    a.step(3)
    for _ in range(3):
        b.step(1)
    assert same(fields(a), fields(b))
    ta, tb = a.thermo(), b.thermo()
    assert (ta.step, ta.temp, ta.status) == (tb.step, tb.temp, 0)
    a.close()
    b.close()


def test_one_type_boxes_alone_same_bits_as_in_a_batch():
    for style, n, kw in ((0, 2500, {}), (0, 20011, dict(exact_rng=1)), (1, 3000, dict(A=25.0, rho_est=0.0)),
                         (1, 20011, dict(A=25.0, rho_est=0.0, exact_rng=1))):
        L = (n / (RHO if style == 0 else 3.0)) ** (1 / 3)
        x, v = lattice(n, L, 3)
        spec = mdpd.box_spec(n, L, style=style, x=x, v=v, seed=9, **kw)
        one, two = mdpd.Batch([spec]), mdpd.Batch([spec, spec])
        for b in (one, two):
            b.setup()
            b.step(25)
            b.step(6)
        assert all(np.array_equal(p, q) for p, q in zip(one.state(0), two.state(1)))
        assert one.thermo(0).nbuild == two.thermo(1).nbuild and one.rebuild_steps() == two.rebuild_steps()
        one.close()
        two.close()


def wall_box(length, wall_rho, exact="fast"):
    """fluid between frozen walls at the low and high x ends"""
    L = np.array([length, 5.0, 5.0])
    rng = np.random.default_rng(4)
    nf, nw = int(6.05 * (L[0] - 4) * 25), int(wall_rho * 4 * 25)
    xf = rng.uniform(0, 1, (nf, 3)) * (L - (4, 0, 0)) + (2, 0, 0)
    xw = rng.uniform(0, 1, (nw, 3)) * (4, 5, 5)
    xw[:, 0] = np.mod(xw[:, 0] - 2, L[0])
    v = np.concatenate([rng.normal(0, 1, (nf, 3)), np.zeros((nw, 3))])
    lam = deck((nf, nw), (0,) * 3, L, "group fluid type 1\ngroup solid type 2",
               "pair_style mdpd/meso 1.0 1.0 77 fluid solid\npair_coeff * * -10 5 4.5 1.0 0.75\n"
               f"pair_modify rng {exact}",
               "fix BC all aboundary/rho/meso cut_rho 0.75 phi_c 0.5 cut_phi 1.0 rho_wall 8.0 wall solid mobile fluid\n"
               "fix NVE fluid nve/meso", np.concatenate([xf, xw]), v)
    return lam, L


# 17 wall particles per unit volume: near-wall rows hold more than the list of wall particles takes
# (n_col2), so the wall fix reads those rows whole
@pytest.mark.parametrize("length,wall_rho", [(12, 8.0), (12, 17.0), (100, 8.0)])
def test_wall_fraction_from_listed_and_whole_rows(length, wall_rho):
    a, L = wall_box(length, wall_rho)
    b, _ = wall_box(length, wall_rho)
    x0 = a.state()[0]
    a.setup()
    b.setup()
    a.step(6)
    for _ in range(6):
        b.step(1)
    assert same(fields(a, FIELDS + ("phi",)), fields(b, FIELDS + ("phi",)))
    a.step(1)
    x, phi, typ = a.field("x"), a.field("phi"), a.field("type")
    tag = a.field("tag")
    w = x[typ == 2]
    assert np.array_equal(w, x0[tag[typ == 2] - 1])  # frozen
    m = np.nonzero(typ == 1)[0]
    d = x[m][:, None, :] - w[None]
    d -= L * np.round(d / L)
    r = np.sqrt((d * d).sum(2))
    want = np.where(r < 1, (1 + 3 * r) * np.clip(1 - r, 0, None) ** 3, 0).sum(1) * 105 / (16 * np.pi * 8.0)
    # a reflected particle (phi above phi_c) has moved since; FP32 coordinates and terms, ~40 of them
    ok = phi[m] <= 0.5
    assert ok.sum() > 0.5 * len(m) and (want > 0.01).sum() > 20
    assert np.abs(phi[m] - want)[ok].max() < 1e-4
    a.close()
    b.close()


def test_tuner_keeps_the_one_launch_runs_of_a_small_box():
    b = mdpd.Batch([mdpd.box_spec(3000, 10.0, style=1, A=25.0, rho_est=0.0, seed=5, init_seed=6)])
    b.setup()
    b.step(5)
    x, v = b.state(0)
    assert b.tune() == (1, 1)
    assert np.array_equal(b.state(0)[0], x) and b.thermo(0).step == 5
    b.step(5)
    assert b.thermo(0).status == 0
    b.close()


def test_small_boxes_stepped_by_several_threads():
    """runs of different boxes from several host threads: each as it is alone"""
    def make(k):
        n = 2500 + 700 * k
        kw = dict(style=1, A=25.0, rho_est=0.0) if k % 2 else {}
        return mdpd.Batch([mdpd.box_spec(n, (n / (3.0 if k % 2 else RHO)) ** (1 / 3), seed=k + 1, init_seed=k + 7, **kw)])

    def go(k, out):
        try:
            b = make(k)
            b.setup()
            for _ in range(6):
                b.step(60)
            out[k] = b.state(0)
            b.close()
        except Exception as e:  # seen by the main thread
            out[k] = e

    alone, together = {}, {}
    for k in range(4):
        go(k, alone)
    th = [threading.Thread(target=go, args=(k, together)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k in range(4):
        assert not isinstance(together[k], Exception), together[k]
        assert same(alone[k], together[k])
