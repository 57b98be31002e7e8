"""The FP64 force and density passes against the oracle where their block plan changes.

A system is cut into blocks by its size and neighbour mode: a warp per atom below 2,400 atoms and in
the stencil and all-pairs modes, 8 lanes an atom above, 4 to 64 atoms a block.  The sizes here sit on
both sides of those lines and leave partly filled blocks, groups and queues; one case has more
neighbours than an atom's queue holds.  Each metal functional has its own arithmetic.  Tolerances
are those of the FP64 path elsewhere: the arithmetic differs from the oracle's by a few roundings
per pair and the order of the sums (forces and energies 1e-12, virial 1e-11 relative).
"""
import numpy as np
import pytest

import oracle
from helpers import FS_FE, FSX_MO, GUPTA_AU, rel_norm_err
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]


def lj(rc_sigma=2.5):
    return "lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {rc_sigma * SIGMA!r}", rc_sigma * SIGMA


def sc(n, m, rc=7.22):
    return "suttonchen", f"e 0.012382 a 3.61 n {n} m {m} c 39.432 cutoff {rc!r}", rc


METALS = {
    "sc96": (sc(9, 6), 3.61, 29), "sc126": (sc(12, 6), 3.61, 29), "sc107": (sc(10, 7), 3.61, 29),
    "sc_real": (sc(9.5, 6.5), 3.61, 29), "fs": (("finnissinclair", FS_FE, 3.569745), 3.6, 26),
    "fsx": (("finnissinclair-ext", FSX_MO, 4.1), 3.6, 42), "gupta": (("gupta", GUPTA_AU, 6.0), 4.08, 79),
}


def crystal(n, a, Z, seed):
    """n atoms of an FCC crystal with some sites removed, displaced by up to 0.2 A."""
    k = 1
    while 4 * k**3 < n:
        k += 1
    pos, L = I.fcc_fast(k, k, k, a)
    pos = I.remove_sites(pos, (len(pos) - n) / len(pos), seed=seed)
    assert len(pos) == n
    return np.mod(I.jitter(pos, 0.2, seed=seed), L), L, np.full(n, Z), np.full(n, 50.0)


def check(pos, L, Z, mass, cm, cm_args, pot):
    name, args, rc = pot
    sim = gbmd.Simulation(len(pos), L)
    sim.set_atoms(pos, Z=Z, mass=mass)
    sim.set_cell_manager(gbmd.Plugin(cm, cm_args))
    sim.add_potential(gbmd.Plugin(name, args))
    sim.update_forces()
    _, _, acc = sim.atoms()
    th = sim.thermo_raw()
    mode = sim.stats()["neighbor_mode"]
    sim.close()
    ref = oracle.PortSim(pos, L, Z, mass, np.zeros_like(pos))
    ref.set_cell_manager(cm, cm_args)
    ref.add_potential(name, args)
    ref.update_forces()
    assert rel_norm_err(acc, ref.atoms()[2]) <= 1e-12
    assert abs(th[1] - ref.energy()) <= 1e-12 * abs(ref.energy())
    assert abs(th[5] - ref.virial()) <= 1e-11 * abs(ref.virial())
    # the stress's trace is the virial
    assert abs(np.trace(th[13:22].reshape(3, 3)) - th[5]) <= 1e-12 * np.abs(th[13:22]).max()
    return mode


@pytest.mark.parametrize("n", [864, 901, 2399, 2400, 2403, 4321])
@pytest.mark.parametrize("cm", ["list", "allpairs", "cells"])
def test_lennard_jones_at_the_edges_of_the_block_plan(n, cm):
    pos, L, Z, mass = crystal(n, 5.6, 18, seed=n)
    name, args, rc = lj()
    if cm == "list":
        c = int(L[0] / rc)
        plugin, cargs = "linkedcell", f"cutoff {rc!r} nx {c} ny {c} nz {c}"
    elif cm == "allpairs":
        plugin, cargs = "minimumimage", f"cutoff {rc!r}"
    else:  # cells narrower than the cutoff, one shell of them: visited exactly as the reference does
        c = int(L[0] / rc) + 1
        plugin, cargs = "linkedcell", f"cutoff {rc!r} nx {c} ny {c} nz {c}"
    mode = check(pos, L, Z, mass, plugin, cargs, (name, args, rc))
    assert mode == {"list": "verlet", "allpairs": "allpairs", "cells": "cells"}[cm]


def test_more_neighbours_than_a_queue_holds():
    pos, L, Z, mass = crystal(5324, 5.26, 18, seed=3)
    _, _, rc = pot = lj(5.0)  # about 440 neighbours, 256 queue entries an atom
    assert check(pos, L, Z, mass, "verletlist", f"cutoff {rc!r} maxneighbors 2000 each 5", pot) == "verlet"


@pytest.mark.parametrize("n", [855, 2911])
@pytest.mark.parametrize("metal", sorted(METALS))
def test_metal_functionals(metal, n):
    pot, a, Z = METALS[metal]
    pos, L, Z, mass = crystal(n, a, Z, seed=n)
    c = max(3, int(L[0] / pot[2] - 1e-9))
    check(pos, L, Z, mass, "linkedcell", f"cutoff {pot[2]!r} nx {c} ny {c} nz {c}", pot)


@pytest.mark.parametrize("cm", ["minimumimage", "linkedcell"])
def test_atoms_outside_the_box(cm):
    """The FP32 pre-test of the stencil and all-pairs modes is a lower bound for any coordinates:
    the reference wraps a distance once, wherever the atoms are."""
    pos, L, Z, mass = crystal(500, 5.6, 18, seed=9)
    pos[::3] += np.array([1.0, 0.0, 1.0]) * L
    pos[1::5] += np.array([0.0, 1.0, 0.0]) * L
    args = f"cutoff {lj()[2]!r}" + ("" if cm == "minimumimage" else " nx 4 ny 4 nz 4")
    check(pos, L, Z, mass, cm, args, lj())
