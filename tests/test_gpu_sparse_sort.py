"""The one-launch sort on grids of more cells than the block cluster has threads (32 cells at a time), and
the chain of kernels beyond its lines by cells: neighbour sets against the oracle (exact multisets), at
build and after steps that rebuild.  A 1,000-atom gas on a million cells is set, sorted and
evaluated in about a millisecond (the one-launch sort took 19)."""
import time

import numpy as np
import pytest

import oracle
from helpers import neighbor_hashes, rel_norm_err
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]
LJ = f"sigma {SIGMA} epsilon {EPS} cutoff 8.5"


def gas(n, cells, seed):
    """n atoms on `cells` cells an axis, on distinct sites 4.4 A apart."""
    L = np.full(3, 9.51 * cells)
    rng = np.random.default_rng(seed)
    m = int(L[0] / 4.4)
    site = rng.choice(m**3, n, replace=False)
    pos = (np.stack([site % m, site // m % m, site // m**2], -1) + 0.5) * (L[0] / m) + rng.uniform(-0.3, 0.3, size=(n, 3))
    return np.mod(pos, L), L, rng


def start(pos, L, vel, precision):
    n = len(pos)
    sim = gbmd.Simulation(n, L)
    sim.set_atoms(pos, vel, Z=np.full(n, 18), mass=np.full(n, 39.948))
    sim.set_cell_manager(gbmd.Plugin("verletlist", "cutoff 8.5 skin 1.0 maxneighbors 400"))
    sim.add_potential(gbmd.Plugin("lennardjones", LJ))
    sim.set_integrator(gbmd.Plugin("velocityverlet", "dt 4.0"))
    sim.set_precision(precision)
    return sim


def reference(pos, L):
    n = len(pos)
    ref = oracle.PortSim(pos, L, np.full(n, 18), np.full(n, 39.948), np.zeros_like(pos))
    ref.set_cell_manager("minimumimage", "cutoff 8.5")
    ref.add_potential("lennardjones", LJ)
    return ref


# one block: up to 32 cells a warp, then more, to 32,768 cells; several blocks to 4,096; then the chain
@pytest.mark.parametrize("n,cells", [(200, 8), (200, 10), (200, 11), (1500, 16), (1500, 31), (700, 32), (700, 33),
                                     (2500, 12), (2500, 16), (2500, 17), (9000, 16)])
def test_neighbours_of_sparse_systems(n, cells):
    pos, L, rng = gas(n, cells, seed=n + cells)
    sim = start(pos, L, rng.normal(size=pos.shape) * 0.01, "fp64")
    sim.update_forces()
    assert np.prod(sim.stats()["cell_grid"]) == cells**3
    for steps in (0, 60):
        if steps:
            sim.do_steps(steps)
            sim.update_forces()
        p, _, acc = sim.atoms()
        ref = reference(p, L)
        counts, idx = sim.neighbors(True, 8.5)
        want, widx = ref.neighbors(True, 8.5)
        np.testing.assert_array_equal(counts, want)
        np.testing.assert_array_equal(neighbor_hashes(counts, idx), neighbor_hashes(want, widx))
        ref.update_forces()
        assert rel_norm_err(acc, ref.atoms()[2]) <= 1e-12
    assert sim.stats()["list_rebuilds"] > 1
    sim.close()


def test_a_gas_on_a_million_cells():
    pos, L, rng = gas(1000, 100, seed=1)
    sim = start(pos, L, rng.normal(size=pos.shape) * 0.01, "mixed")

    def call():
        sim.set_atoms(pos, Z=np.full(1000, 18), mass=np.full(1000, 39.948))
        sim.update_forces()

    call()
    t = []
    for _ in range(5):
        a = time.perf_counter()
        call()
        t.append(time.perf_counter() - a)
    assert min(t) < 0.006, t
    sim.close()
