"""A mixed system's whole record -- positions, velocities, accelerations and all 22 thermo fields -- is the
same bit for bit whatever the lanes per atom, so also in a batch whose size asks for other lanes than the
system alone would get.

The sums that lanes could group otherwise are the kinetic ones (FP64 over 32 consecutive atoms) and stress
(FP32 over an atom's list).  Sizes leave partly filled blocks; the copper's cutoff lies on a shell, so that
guard-band pairs are added to the stress sums after the list, one or several an atom (without thermal
motion all of them).
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


def crystal(n, a, seed, jitter=0.05):
    k = 1
    while 4 * k**3 < n:
        k += 1
    pos, L = I.fcc_fast(k, k, k, a)
    pos = I.remove_sites(pos, (len(pos) - n) / len(pos), seed=seed)
    if jitter:
        pos = I.jitter(pos, jitter, seed=seed)
    m = np.full(n, 60.0)
    return np.mod(pos, L), I.maxwell_boltzmann(m, 300.0, seed=seed), m, L


def run(systems, pot, steps, lanes=()):
    name, args, rc, _, Z = pot
    b = gbmd.Batch([len(s[0]) for s in systems], [s[3] for s in systems])
    for k, (pos, vel, m, _) in enumerate(systems):
        b.set_atoms(k, pos, vel, Z=Z, mass=m)
    b.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin 0.4 maxneighbors 400"))
    b.add_potential(gbmd.Plugin(name, args))
    b.set_integrator(gbmd.Plugin("velocityverlet", "dt 2.0"))
    b.set_precision("mixed")
    for ln in lanes:
        b.set_option("lanes_per_atom", ln)
    b.update_forces()
    first = b.thermo(0)["raw"]
    b.do_steps(steps)
    out = (*b.atoms(0), first, b.thermo(0)["raw"])
    b.close()
    return out


def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# 8 lanes to 9,728 atoms, 4 to 38,912, 2 to 77,824 (8 blocks on each of 152 SMs), then one
@pytest.mark.parametrize("kind,n", [(k, n) for k in sorted(POTS) for n in (1001, 10037)] + [("lj", 39100), ("sc", 39100)])
@pytest.mark.parametrize("jitter", [0.05, 0.0])
def test_record_alone_and_beside_a_large_system(kind, n, jitter):
    pot = POTS[kind]
    small = crystal(n, pot[3], seed=n % 97, jitter=jitter)
    filler = crystal(80001, pot[3], seed=5)  # more than 77,824 atoms: a single lane for every system
    same(run([small], pot, 13), run([small, filler], pot, 13))


@pytest.mark.parametrize("lanes", [2, 4, 8, 16, 32])
def test_record_by_lanes(lanes):
    systems = [crystal(n, POTS["lj"][3], seed=n) for n in (1001, 333)]
    same(run(systems, POTS["lj"], 13, [lanes]), run(systems, POTS["lj"], 13, [1]))


def test_lanes_by_size_again():
    """0 gives the choice back to the engine; other numbers stay refused."""
    small = crystal(1001, POTS["lj"][3], seed=3)
    same(run([small], POTS["lj"], 13, [32, 0]), run([small], POTS["lj"], 13))
    for ln in (3, 64, -1):
        with pytest.raises(gbmd.GbmdError, match="lanes_per_atom"):
            run([small], POTS["lj"], 1, [ln])


@pytest.mark.parametrize("n", [1500, 12000])
def test_record_with_species_filters(n):
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
        out.append((*sim.atoms(), sim.thermo()["raw"]))
        sim.close()
    same(*out)


def test_lanes_follow_the_active_systems():
    """A large system that retires leaves the small one with the lanes it gets alone, and the same record."""
    small, filler = crystal(4001, POTS["lj"][3], seed=2), crystal(80001, POTS["lj"][3], seed=5)
    _, args, rc, _, Z = POTS["lj"]
    out = []
    for systems in ([small], [small, filler]):
        b = gbmd.Batch([len(s[0]) for s in systems], [s[3] for s in systems])
        for k, (pos, vel, m, _) in enumerate(systems):
            b.set_atoms(k, pos, vel, Z=Z, mass=m)
        b.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin 0.4 maxneighbors 400"))
        b.add_potential(gbmd.Plugin("lennardjones", args))
        b.set_integrator(gbmd.Plugin("velocityverlet", "dt 2.0"))
        b.set_precision("mixed")
        b.update_forces()
        b.do_steps(3)
        if len(systems) > 1:
            b.set_active(1, False)
        b.do_steps(20)
        out.append((*b.atoms(0), b.thermo(0)["raw"]))
        b.close()
    same(*out)


@pytest.mark.parametrize("lanes", [2, 4, 8, 16, 32])
def test_record_beyond_the_fixed_point_range(lanes):
    """Two atoms 0.001 A apart: sums that leave FP32's range are the same nonsense in every lane count."""
    pos, vel, m, L = crystal(333, POTS["lj"][3], seed=9)
    pos[200] = pos[100] + 0.0005
    system = [(pos, vel, m, L)]
    same(run(system, POTS["lj"], 0, [lanes])[3:], run(system, POTS["lj"], 0, [1])[3:])
