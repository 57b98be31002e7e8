"""Which pairs the FP64 passes take, where the FP32 pre-test of a candidate and the reference's cutoff
test look at different distances.

The reference wraps a difference of coordinates once, wherever the atoms are.  The list's FP32 offsets
see the nearest image.  Positions are not folded into the box when they are set, and atoms with a fixed
position never are, so the two differ by box lengths.  Tolerances are those of the FP64 path elsewhere:
forces and energies 1e-12, virial 1e-11 relative.
"""
import numpy as np
import pytest

import oracle
from helpers import FS_FE, SC_CU, rel_norm_err
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]
RC = 2.5 * SIGMA
POTS = {"lj": ("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {RC!r}", RC, 5.6, 18),
        "sc": ("suttonchen", SC_CU, 7.22, 3.61, 29), "fs": ("finnissinclair", FS_FE, 3.569745, 3.6, 26)}


def crystal(n, a, seed):
    """n atoms of an FCC crystal with some sites removed, displaced by up to 0.2 A."""
    k = 1
    while 4 * k**3 < n:
        k += 1
    pos, L = I.fcc_fast(k, k, k, a)
    pos = I.remove_sites(pos, (len(pos) - n) / len(pos), seed=seed)
    return np.mod(I.jitter(pos, 0.2, seed=seed), L), L


def pair_of(pos, L, pot, cm, cm_args, Z=18, mass=50.0, vel=None, flags=None):
    """The same system in libgbmd (FP64) and in the oracle, forces evaluated."""
    n = len(pos)
    Z, mass = np.full(n, Z), np.full(n, mass)
    vel = np.zeros_like(pos) if vel is None else vel
    sim = gbmd.Simulation(n, L)
    sim.set_atoms(pos, vel, Z=Z, mass=mass)
    ref = oracle.PortSim(pos, L, Z, mass, vel, flags=flags)
    if flags is not None:
        sim.set_flags(flags)
    for s in (sim, ref):
        if s is sim:
            s.set_cell_manager(gbmd.Plugin(cm, cm_args))
            s.add_potential(gbmd.Plugin(*pot))
            s.set_integrator(gbmd.Plugin("velocityverlet", "dt 1.0"))
        else:
            s.set_cell_manager(cm, cm_args)
            s.add_potential(*pot)
            s.set_integrator(1.0)
        s.update_forces()
    return sim, ref


def agree(sim, ref, tol=1e-12):
    assert rel_norm_err(sim.atoms()[2], ref.atoms()[2]) <= tol
    th = sim.thermo_raw()
    assert abs(th[1] - ref.energy()) <= tol * abs(ref.energy())
    assert abs(th[5] - ref.virial()) <= 10 * tol * abs(ref.virial())


def list_manager(cm, rc, L):
    if cm == "verletlist":
        return f"cutoff {rc!r} maxneighbors 400 each 5"
    c = int(L[0] / rc)  # cells at least as wide as the cutoff
    return f"cutoff {rc!r} nx {c} ny {c} nz {c}"


@pytest.mark.parametrize("cm", ["verletlist", "linkedcell"])
@pytest.mark.parametrize("kind,n", [("lj", 500), ("lj", 2500), ("sc", 864), ("sc", 2903), ("fs", 500)])
def test_list_pairs_of_atoms_a_box_length_outside(kind, n, cm):
    name, args, rc, a, Z = POTS[kind]
    pos, L = crystal(n, a, seed=n)
    pos[::3] += np.array([1.0, 0.0, 1.0]) * L
    pos[1::5] += np.array([0.0, 1.0, 0.0]) * L
    sim, ref = pair_of(pos, L, (name, args), cm, list_manager(cm, rc, L), Z=Z)
    assert sim.stats()["neighbor_mode"] == "verlet"
    agree(sim, ref)
    sim.close()


def test_a_fixed_atom_outside_the_box_over_steps():
    name, args, rc, a, Z = POTS["lj"]
    pos, L = crystal(500, a, seed=4)
    pos[7] += L
    pos[123] += np.array([0.0, 0.0, 1.0]) * L
    flags = np.zeros(500, dtype=np.uint8)
    flags[[7, 123]] = 2  # fixed position
    vel = I.maxwell_boltzmann(np.full(500, 50.0), 100.0, seed=4)
    vel[[7, 123]] = 0.0
    sim, ref = pair_of(pos, L, (name, args), "verletlist", list_manager("verletlist", rc, L), vel=vel, flags=flags)
    agree(sim, ref)
    sim.do_steps(5)
    ref.do_steps(5)
    assert sim.stats()["neighbor_mode"] == "verlet"
    assert np.array_equal(sim.atoms()[0][[7, 123]], pos[[7, 123]])
    agree(sim, ref, 1e-11)  # five steps pass the forces' rounding on
    sim.close()
