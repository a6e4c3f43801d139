"""Launch shapes that depend on the size of the work: every shape gives the same bits, and the
smallest one agrees with the FP64 oracle engine."""
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
