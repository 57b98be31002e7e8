"""Which pairs the FP64 passes take, where the FP32 pre-test of a candidate and the reference's cutoff
test look at different distances.

The reference wraps a difference of coordinates once, wherever the atoms are.  The list's FP32 offsets
see the nearest image.  Positions are not folded into the box when they are set, and atoms with a fixed
position never are, so the two differ by box lengths; and a list on the `each` clock alone outlives the images
that it was built with.  Tolerances are those of the FP64 path elsewhere:
forces and energies 1e-12, virial 1e-11 relative.
"""
import numpy as np
import pytest

import oracle
from helpers import FS_FE, FSX_MO, GUPTA_AU, SC_CU, rel_norm_err
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
    snapshot = sim.checkpoint()
    sim.do_steps(12)
    other, _ = pair_of(pos, L, (name, args), "verletlist", list_manager("verletlist", rc, L), vel=vel, flags=flags)
    other.restore(snapshot)
    other.do_steps(12)
    for a, b in zip(sim.atoms(), other.atoms()):
        np.testing.assert_array_equal(a, b)
    other.close()
    sim.close()


def test_a_list_that_outlives_its_images():
    """Layers sliding along x for longer than the list is valid: pairs listed through one image come
    inside through the other, which the reference, wrapping afresh, then takes."""
    L = np.full(3, 20.0)
    k = np.arange(4) * 5.0
    pos = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    odd = (pos[:, 1] / 5.0).astype(int) % 2 == 1
    pos[odd, 0] += 2.6
    pos = np.mod(I.jitter(pos, 0.1, seed=3), L)
    vel = np.zeros_like(pos)
    vel[:, 0] = np.where(odd, 0.04, -0.04)
    rc = 8.5
    pot = ("lennardjones", f"sigma 3.405 epsilon 0.0103 cutoff {rc}")
    sim, ref = pair_of(pos, L, pot, "verletlist", "cutoff 8.5 maxneighbors 400 each 100000", mass=1000.0, vel=vel)
    # the same list without libgbmd's own rebuild on displacement
    sim.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff 8.5 skin {0.08 * rc!r} maxneighbors 400 each 100000 rebuild each"))
    sim.update_forces()
    agree(sim, ref)
    before = sim.stats()["list_rebuilds"]
    sim.do_steps(80)
    ref.do_steps(80)
    assert sim.stats()["list_rebuilds"] == before and sim.stats()["neighbor_mode"] == "verlet"
    agree(sim, ref, 1e-11)
    sim.close()


def test_coordinates_many_box_lengths_outside():
    """Pairs within 3e-5 of the cutoff, five box lengths up: FP32 offsets resolve 1e-4 A there."""
    L = np.full(3, 400.0)
    k = 12.0 + 25.0 * np.arange(15)
    first = np.stack(np.meshgrid(k, k[:5], k[:4], indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(5)
    u = rng.normal(size=first.shape)
    u /= np.linalg.norm(u, axis=1)[:, None]
    second = first + u * (RC * (1.0 + np.linspace(-3e-5, 3e-5, len(first))))[:, None]
    pos = np.concatenate([first, second]) + 5.0 * L
    name, args, rc, _, _ = POTS["lj"]
    sim, ref = pair_of(pos, L, (name, args), "verletlist", list_manager("verletlist", rc, L))
    assert sim.stats()["neighbor_mode"] == "verlet"
    agree(sim, ref)
    sim.close()


@pytest.mark.parametrize("cm", ["minimumimage", "verletlist"])
@pytest.mark.parametrize("kind", ["gupta", "fs", "fsx", "sc", "sc126", "sc107"])
def test_coincident_atoms_spoil_only_themselves(kind, cm):
    """r = 0 is a distance like any other to the densities of Gupta and Finnis-Sinclair metals, and an
    infinite density (no embedding factor) to Sutton-Chen: only the two atoms' forces are undefined."""
    name, args, rc, a, Z = {
        "gupta": ("gupta", GUPTA_AU, 6.0, 4.08, 79), "fs": ("finnissinclair", FS_FE.replace("B 1.8", "B 0.5"), 3.569745, 3.6, 26),
        "fsx": ("finnissinclair-ext", FSX_MO, 4.1, 3.6, 42),
        "sc": POTS["sc"], "sc126": ("suttonchen", "e 0.02 a 4.09 n 12 m 6 c 144.4 cutoff 8.18", 8.18, 4.09, 47),
        "sc107": ("suttonchen", "e 0.012 a 3.61 n 10 m 7 c 39.4 cutoff 7.22", 7.22, 3.61, 29)}[kind]
    pos, L = crystal(864, a, seed=8)
    pos[300] = pos[301]
    cm_args = f"cutoff {rc!r}" if cm == "minimumimage" else list_manager(cm, rc, L)
    sim, ref = pair_of(pos, L, (name, args), cm, cm_args, Z=Z)
    got, want = sim.atoms()[2], ref.atoms()[2]
    rest = np.delete(np.arange(len(pos)), [300, 301])
    assert np.isnan(got[[300, 301]]).all() and np.isnan(want[[300, 301]]).all()
    assert np.isfinite(want[rest]).all()
    assert rel_norm_err(got[rest], want[rest]) <= 1e-12
    np.testing.assert_allclose(sim.thermo_raw()[1], ref.energy(), rtol=1e-12)  # NaN where the reference's is
    sim.close()


@pytest.mark.parametrize("cm,cm_args", [("minimumimage", "cutoff 8.5"), ("linkedcell", "cutoff 8.5 nx 4 ny 4 nz 4"),
                                        ("verletlist", "cutoff 8.5 maxneighbors 400 each 5")])
def test_no_pair_is_inside_a_cutoff_that_is_not_a_number(cm, cm_args):
    pos, L = crystal(500, 5.6, seed=6)
    sim, ref = pair_of(pos, L, ("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff nan"), cm, cm_args)
    assert not ref.atoms()[2].any() and not sim.atoms()[2].any() and sim.thermo_raw()[1] == 0.0
    sim.close()


def test_cells_of_atoms_one_box_length_below():
    """The reference's WrapAround takes cell -n to cell n: along x and y that is the first cell of the next
    row or plane, which the stencil mode, visiting cells as the reference does, keeps to."""
    name, args, rc, a, _ = POTS["lj"]
    pos, L = crystal(500, a, seed=12)
    d = L / 4
    low = pos < d
    pos[low[:, 0] & (pos[:, 2] < 3 * d[2])] -= np.array([1.0, 0.0, 0.0]) * L
    pos[low[:, 1] & (pos[:, 2] < 3 * d[2]) & (pos[:, 0] > 0)] -= np.array([0.0, 1.0, 0.0]) * L
    assert (pos < 0).any(axis=0).tolist() == [True, True, False]
    sim, ref = pair_of(pos, L, (name, args), "linkedcell", f"cutoff {rc!r} nx 4 ny 4 nz 4")
    assert sim.stats()["neighbor_mode"] == "cells"
    agree(sim, ref)
    sim.close()
