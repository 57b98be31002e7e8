"""Kernel-class times cover the steps of integrators that otherwise run as captured blocks."""
import pytest

from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")


@pytest.mark.parametrize("integrator", ["beeman", "leapfrog"])
def test_every_force_evaluation_is_timed(integrator):
    w = I.lj_system(5, 0.8, 1.0, seed=3)
    rc = 2.5 * I.LJ_AR["sigma"]
    sim = gbmd.Simulation(w["natoms"], w["L"])
    sim.set_atoms(w["pos"], w["vel"], Z=w["Z"], mass=w["mass"])
    sim.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} maxneighbors 256"))
    sim.add_potential(gbmd.Plugin("lennardjones", f"sigma {I.LJ_AR['sigma']} epsilon {I.LJ_AR['epsilon']} cutoff {rc!r}"))
    sim.set_integrator(gbmd.Plugin(integrator, "dt 1.0"))
    sim.set_precision("mixed")
    sim.update_forces()
    sim.set_option("time_kernels", 1)
    before = sim.stats()["force_launches"]
    sim.do_steps(45)
    assert sim.stats()["force_launches"] - before >= 45
