"""Captured steps of batches on both sides of the line between a conditional rebuild (up to 8 active
systems) and the chain in line: bit for bit the directly launched steps, with systems that rebuild at
their own times and one that retires on the way."""
import numpy as np
import pytest

from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]


@pytest.mark.parametrize("count", [2, 8, 9])
def test_captured_batches_equal_direct_steps(count):
    # 2,916 atoms: past the one-launch sort of a batch
    systems = [I.lj_system(9 if k == 0 else 4 + k % 3, 0.8, 0.05 + 0.4 * k, seed=60 + k) for k in range(count)]
    rc = 2.5 * SIGMA
    out = []
    for mode in (0, 2):
        b = gbmd.Batch([s["natoms"] for s in systems], [s["L"] for s in systems])
        for k, s in enumerate(systems):
            b.set_atoms(k, s["pos"], s["vel"], Z=s["Z"], mass=s["mass"])
        b.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin {0.2 * SIGMA!r} maxneighbors 256"))
        b.add_potential(gbmd.Plugin("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {rc!r}"))
        b.set_integrator(gbmd.Plugin("velocityverlet", "dt 10.0"))
        b.set_precision("mixed")
        b.set_option("graph_mode", mode)
        b.update_forces()
        b.do_steps(31)
        b.set_active(count - 1, False)
        b.do_steps(30)
        out.append([x for k in range(count) for x in (*b.atoms(k), b.thermo(k)["raw"])] + [b.stats()["list_rebuilds"]])
        b.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    assert out[0][-1] > 2 * count
