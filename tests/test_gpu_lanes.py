"""The mixed passes with several lanes per atom (chosen for systems that do not fill the GPU) against
one lane per atom.

The lane count follows the atoms of all systems of an engine, so a small system alone runs with 8, 4
or 2 lanes and beside a large one with a single lane.  Every group of list entries is summed alike and
the partials are integers: positions, velocities, accelerations, energies and virials are equal bit
for bit; stress sums are FP32 per lane (1e-6 relative to the largest component).  Sizes leave partly
filled blocks of 16, 32 and 64 atoms; the copper's cutoff lies on a shell, so that many pairs are
decided in the guard band.
"""
import numpy as np
import pytest

from helpers import FS_FE, GUPTA_AU, SC_CU
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]
LJ = f"sigma {SIGMA} epsilon {EPS} cutoff {2.5 * SIGMA!r}"
POTS = {"lj": ("lennardjones", LJ, 8.5125, 5.6, 18), "sc": ("suttonchen", SC_CU, 7.22, 3.61, 29),
        "sc126": ("suttonchen", "e 0.02 a 4.09 n 12 m 6 c 144.4 cutoff 8.18", 8.18, 4.09, 47),
        "fs": ("finnissinclair", FS_FE, 3.569745, 3.6, 26), "gupta": ("gupta", GUPTA_AU, 6.0, 4.08, 79)}


def crystal(n, a, seed):
    k = 1
    while 4 * k**3 < n:
        k += 1
    pos, L = I.fcc_fast(k, k, k, a)
    pos = I.remove_sites(pos, (len(pos) - n) / len(pos), seed=seed)
    pos = np.mod(I.jitter(pos, 0.05, seed=seed), L)
    m = np.full(n, 60.0)
    return pos, I.maxwell_boltzmann(m, 300.0, seed=seed), m, L


def run(systems, pot, steps):
    name, args, rc, _, Z = pot
    b = gbmd.Batch([len(s[0]) for s in systems], [s[3] for s in systems])
    for k, (pos, vel, m, _) in enumerate(systems):
        b.set_atoms(k, pos, vel, Z=Z, mass=m)
    b.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin 0.4 maxneighbors 400"))
    b.add_potential(gbmd.Plugin(name, args))
    b.set_integrator(gbmd.Plugin("velocityverlet", "dt 2.0"))
    b.set_precision("mixed")
    b.update_forces()
    b.do_steps(steps)
    out = b.atoms(0), b.thermo(0)
    b.close()
    return out


# 8 lanes to 9,728 atoms, 4 to 38,912, 2 to 77,824 (8 blocks on each of 152 SMs), then one
@pytest.mark.parametrize("n", [1001, 9700, 10037, 38801, 39100, 77777])
@pytest.mark.parametrize("kind", sorted(POTS))
def test_lanes_equal_one_lane(kind, n):
    pot = POTS[kind]
    if kind != "lj" and n > 20000 and kind != "sc":
        pytest.skip("the larger sizes with two functionals are enough")
    small = crystal(n, pot[3], seed=n % 97)
    filler = crystal(80001, pot[3], seed=5)  # more than 77,824 atoms: a single lane for every system
    (a, ta), (b, tb) = run([small], pot, 13), run([small, filler], pot, 13)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    assert ta["potential_energy"] == tb["potential_energy"]
    assert ta["virial"] == tb["virial"]
    np.testing.assert_allclose(ta["raw"][2:9], tb["raw"][2:9], rtol=1e-11, atol=1e-11 * abs(tb["raw"][2]))
    np.testing.assert_allclose(ta["stress"], tb["stress"], rtol=0, atol=1e-6 * np.abs(tb["stress"]).max())


@pytest.mark.parametrize("n", [1500, 12000])
def test_lanes_with_species_filters(n):
    """Several potentials with species filters: the passes carry their partial sums on."""
    pos, vel, m, L = crystal(n, 5.6, seed=7)
    Z = np.where(np.arange(n) % 3 == 0, 36, 18).astype(np.int32)
    out = []
    for lanes in (0, 1):
        sim = gbmd.Simulation(n, L)
        sim.set_atoms(pos, vel, Z=Z, mass=m)
        sim.set_cell_manager(gbmd.Plugin("verletlist", "cutoff 8.5 skin 0.6 maxneighbors 400"))
        for args, s1, s2 in (("sigma 3.405 epsilon 0.0103 cutoff 8.5", 18, 18), ("sigma 3.6 epsilon 0.014 cutoff 8.0", 36, 36),
                             ("sigma 3.5 epsilon 0.012 cutoff 8.2", 18, 36)):
            sim.add_potential(gbmd.Plugin("lennardjones", args), s1, s2)
        sim.set_integrator(gbmd.Plugin("velocityverlet", "dt 2.0"))
        sim.set_precision("mixed")
        if lanes:
            sim.set_option("lanes_per_atom", lanes)
        sim.update_forces()
        sim.do_steps(13)
        out.append((sim.atoms(), sim.thermo()))
        sim.close()
    for x, y in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(x, y)
    assert out[0][1]["potential_energy"] == out[1][1]["potential_energy"]
    assert out[0][1]["virial"] == out[1][1]["virial"]
