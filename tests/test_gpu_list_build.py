"""The two list builders against the oracle where their shapes change: thin and crowded cells, a
stencil beyond the staged run, rows too long for shared memory, grids on both sides of the line
between a block and a warp per cell, and batches of which only some systems rebuild.

Neighbour sets are exact (multisets); sums as for the FP64 path elsewhere (1e-12)."""
import numpy as np
import pytest

import oracle
from helpers import neighbor_hashes, rel_norm_err
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]


def crystal(k, drop, seed, a=5.6, jitter=0.3):
    pos, L = I.fcc_fast(k, k, k, a)
    pos = I.remove_sites(pos, drop / len(pos), seed=seed)
    return np.mod(I.jitter(pos, jitter, seed=seed), L), L


def sims(pos, L, rc, cm_args):
    n = len(pos)
    Z, mass = np.full(n, 18), np.full(n, 39.948)
    pot = f"sigma {SIGMA} epsilon {EPS} cutoff {rc!r}"
    sim = gbmd.Simulation(n, L)
    sim.set_atoms(pos, Z=Z, mass=mass)
    sim.set_cell_manager(gbmd.Plugin("verletlist", cm_args))
    sim.add_potential(gbmd.Plugin("lennardjones", pot))
    ref = oracle.PortSim(pos, L, Z, mass, np.zeros_like(pos))
    ref.set_cell_manager("minimumimage", f"cutoff {rc!r}")
    ref.add_potential("lennardjones", pot)
    return sim, ref


# cutoff (A), cells per edge, removed sites: cells of about 3, 15, 60 and 330 atoms (the last with
# 9,000 in the stencil), and 17^3 = 4,913 cells (a warp each)
@pytest.mark.parametrize("rc, k, drop", [(4.6, 8, 5), (8.5, 8, 0), (13.4, 9, 31), (23.0, 10, 7), (4.8, 16, 100)])
@pytest.mark.parametrize("stencil", [1, 2])
def test_neighbour_sets(rc, k, drop, stencil):
    pos, L = crystal(k, drop, seed=k)
    sim, ref = sims(pos, L, rc, f"cutoff {rc!r} skin 0.4 maxneighbors 4000")
    sim.set_option("stencil", stencil)
    counts, idx = sim.neighbors(True, rc)
    want, widx = ref.neighbors(True, rc)
    np.testing.assert_array_equal(counts, want)
    np.testing.assert_array_equal(neighbor_hashes(counts, idx), neighbor_hashes(want, widx))


def test_rows_too_long_for_shared_memory():
    pos, L = crystal(14, 0, seed=2)
    sim, ref = sims(pos, L, 36.0, "cutoff 36.0 skin 2.9 maxneighbors 9000")
    sim.update_forces()
    ref.update_forces()
    assert sim.stats()["list_capacity"] > 7168
    assert rel_norm_err(sim.atoms()[2], ref.atoms()[2]) <= 1e-12
    assert abs(sim.thermo_raw()[1] - ref.energy()) <= 1e-12 * abs(ref.energy())


def test_systems_of_a_batch_rebuild_at_their_own_times():
    """Hot and cold systems of several sizes, so that most steps rebuild some of them only."""
    systems = [I.lj_system(k, 0.8, t, seed=90 + k) for k, t in ((4, 2.0), (5, 0.1), (9, 1.5), (6, 0.01), (7, 0.8))]
    rc = 2.5 * SIGMA

    def run(obj, atoms, which):
        for s, w in enumerate(which):
            atoms(s, w)
        obj.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin {0.2 * SIGMA!r} maxneighbors 256"))
        obj.add_potential(gbmd.Plugin("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {rc!r}"))
        obj.set_integrator(gbmd.Plugin("velocityverlet", "dt 10.0"))
        obj.set_precision("mixed")
        obj.update_forces()
        obj.do_steps(47)

    b = gbmd.Batch([w["natoms"] for w in systems], [w["L"] for w in systems])
    run(b, lambda s, w: b.set_atoms(s, w["pos"], w["vel"], Z=w["Z"], mass=w["mass"]), systems)
    total = 0
    for s, w in enumerate(systems):
        sim = gbmd.Simulation(w["natoms"], w["L"])
        run(sim, lambda _, x: sim.set_atoms(x["pos"], x["vel"], Z=x["Z"], mass=x["mass"]), [w])
        for x, y in zip(b.atoms(s), sim.atoms()):
            np.testing.assert_array_equal(x, y)
        total += sim.stats()["list_rebuilds"]
    assert b.stats()["list_rebuilds"] == total
