"""Captured blocks of the integrators other than velocity Verlet: bit for bit the directly launched steps,
over calls of odd and even numbers of steps, a change of dt and of the thermostat's target between captured
calls, and a snapshot."""
import numpy as np
import pytest

from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]
INTEGRATORS = ["euler", "leapfrog", "verlet", "beeman", "nosehoover"]


def integrator(name, dt, t):
    return gbmd.Plugin(name, f"dt {dt}" + (f" fmass 2e9 t {t}" if name == "nosehoover" else ""))


@pytest.mark.parametrize("name", INTEGRATORS)
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_captured_steps_equal_direct_steps(name, precision):
    s = I.lj_system(6, 0.8, 1.2, seed=17)
    rc = 2.5 * SIGMA
    dt = 0.2 if name == "euler" else 4.0
    out = []
    for mode in (0, 2):
        sim = gbmd.Simulation(s["natoms"], s["L"])
        sim.set_atoms(s["pos"], s["vel"], Z=s["Z"], mass=s["mass"])
        sim.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin {0.2 * SIGMA!r} maxneighbors 256"))
        sim.add_potential(gbmd.Plugin("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {rc!r}"))
        sim.set_integrator(integrator(name, dt, 120.0))
        sim.set_precision(precision)
        sim.set_option("graph_mode", mode)
        sim.update_forces()
        rec = []
        for n in (25, 40, 7, 33):
            sim.do_steps(n)
            rec += [*sim.atoms(), sim.thermo_raw()]
        sim.set_integrator(integrator(name, 0.5 * dt, 90.0))
        sim.do_steps(41)
        rec += [*sim.atoms(), sim.thermo_raw()]
        ck = sim.checkpoint()
        sim.do_steps(23)
        rec += [*sim.atoms(), sim.thermo_raw()]
        sim.restore(ck)
        sim.do_steps(23)
        rec += [*sim.atoms(), sim.thermo_raw(), sim.thermo_log(), sim.stats()["list_rebuilds"]]
        out.append(rec)
        sim.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    for x, y in zip(out[0][20:24], out[0][24:28]):  # the restored run is the run
        np.testing.assert_array_equal(x, y)


def test_a_target_set_between_captured_calls_counts():
    """Nose-Hoover with another target after the capture: the friction follows the new one."""
    s = I.lj_system(6, 0.8, 1.2, seed=18)
    rc = 2.5 * SIGMA
    out = []
    for t in (120.0, 900.0):
        sim = gbmd.Simulation(s["natoms"], s["L"])
        sim.set_atoms(s["pos"], s["vel"], Z=s["Z"], mass=s["mass"])
        sim.set_cell_manager(gbmd.Plugin("verletlist", f"cutoff {rc!r} skin {0.3 * SIGMA!r} maxneighbors 256"))
        sim.add_potential(gbmd.Plugin("lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {rc!r}"))
        sim.set_integrator(integrator("nosehoover", 4.0, 120.0))
        sim.update_forces()
        sim.do_steps(40)
        sim.set_integrator(integrator("nosehoover", 4.0, t))
        sim.do_steps(40)
        out.append(sim.thermo()["kinetic_energy"])
        sim.close()
    assert out[0] != out[1]
