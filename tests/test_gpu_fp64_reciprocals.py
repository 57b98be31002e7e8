"""The FP64 passes' reciprocal and reciprocal square root (one third-order step from the hardware's
approximation) against exact rational arithmetic, through the energies of pairs of atoms, one pair a
system.

u = 2^-53.  1/sqrt: the step's e is off by u (rounding of x y), half of which reaches the result, which is
rounded once, and the neglected term is 2^-60: at most 1.6 u, tested at 2 u.  A Sutton-Chen pair with
n = 1, a = e = 1 and no embedding has just this energy.  1/x: e is exact but for its own rounding (2^-73):
1.02 u.  Lennard-Jones with sigma = 2, epsilon = 1/4 has the energy x^6 - x^3, x = 4 / r^2: 3.1 u from the
reciprocal and 2 u from the products in x^3, twice that where x^6 dominates, one rounding for the bracket
and one for the product: at most 13 u, tested at 14 u away from the zero of the bracket.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")

U = Fraction(1, 2**53)


def pair_energies(r, pot):
    b = gbmd.Batch([2] * len(r), [np.full(3, 512.0)] * len(r))
    for k, x in enumerate(r):
        b.set_atoms(k, np.array([[0.0, 0.0, 0.0], [x, 0.0, 0.0]]), np.zeros((2, 3)), Z=np.full(2, 18), mass=np.full(2, 40.0))
    b.set_cell_manager(gbmd.Plugin("minimumimage", "cutoff 250"))
    b.add_potential(gbmd.Plugin(*pot))
    b.set_precision("fp64")
    b.update_forces()
    e = [b.thermo(k)["potential_energy"] for k in range(len(r))]
    b.close()
    return e


def distances(lo, hi, n, seed):
    return np.exp(np.random.default_rng(seed).uniform(np.log(lo), np.log(hi), n))


def test_reciprocal_square_root():
    r = distances(2e-3, 240.0, 700, 1)
    for x, e in zip(r, pair_energies(r, ("suttonchen", "e 1 a 1 n 1 m 6 c 0 cutoff 250"))):
        # (e - 1/sqrt(r2)) / (1/sqrt(r2)) from e^2 r2 = (1 + d)^2: d = (e^2 r2 - 1) / 2, to first order
        d = (Fraction(e) ** 2 * Fraction(x * x) - 1) / 2
        assert abs(d) <= 2 * U, (x, float(d / U))


def test_reciprocal():
    r = np.concatenate([distances(2e-3, 1.6, 350, 2), distances(2.5, 240.0, 350, 3)])
    for x, e in zip(r, pair_energies(r, ("lennardjones", "sigma 2 epsilon 0.25 cutoff 250"))):
        x3 = (4 / Fraction(x * x)) ** 3
        d = Fraction(e) / (x3 * x3 - x3) - 1
        assert abs(d) <= 14 * U, (x, float(d / U))
