"""Classic DPD with a weight exponent other than 1, for pairs at the cutoff."""
import numpy as np
import pytest

import mdpd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [0.7, 0.9, 1.13])  # 1 - r / cut rounds below 0 for the last r below each
@pytest.mark.parametrize("expw", [0.5, 2.0])
def test_pairs_just_inside_the_cutoff(cut, expw):
    """16 isolated pairs 0 to 15 FP32 steps inside the cutoff: their weights are those of the cutoff, 0 to
    within rounding, and their forces finite"""
    f = np.float32
    d, cutsq = f(cut) * f(1.000001), f(cut * cut)
    while not f(d * d) < cutsq:
        d = np.nextafter(d, f(0))
    x = []
    for k in range(16):
        y, z = 1.5 + 3 * (k % 4), 1.5 + 3 * (k // 4)
        x += [(6.0, y, z), (6.0 - float(d), y, z)]  # exact in FP32 about the box's centre
        d = np.nextafter(d, f(0))
    x = np.array(x)
    lam = mdpd.Lammps()
    lam.commands(f"""units lj
boundary p p p
neighbor 0.3 bin
neigh_modify every 1 delay 0 check yes
atom_style dpd/atomic/meso 8
region box block 0 12 0 12 0 12 units box
create_box 1 box
create_atoms 1 random {len(x)} 11 box
mass 1 1
pair_style dpd/meso {cut} 77
pair_coeff 1 1 25 4.5 3.0 {expw} {cut}
fix NVE all nve/meso
timestep 0.01
run_style mvv/meso""")
    lam.set_state(x, np.zeros_like(x))
    lam.setup()
    force = lam.field("force")[:, :3]
    # (16 + 1 steps of 2^-24 of the cutoff's binade) / cut < 2.5e-6 = w; sigma w^0.5 |gaussian| / sqrt(dt) with
    # |gaussian| <= 4, and A w
    assert np.isfinite(force).all() and np.abs(force).max() < 3 * 2.5e-6 ** 0.5 * 4 * 10 + 25 * 2.5e-6
    lam.step(2)
    assert lam.thermo().status == 0 and np.isfinite(lam.field("v")).all()
    lam.close()
