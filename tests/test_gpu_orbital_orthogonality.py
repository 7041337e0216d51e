"""Orthogonality of the occupied orbitals, seen in the density they give: with every occupation 2 or 0
(electronic temperature 0) P S P = 2 P exactly, and two orbitals that overlap by x leave 4 x there.

Tolerance: two vectors of the tridiagonal overlap by the rounding of their factorisations, eps |T| over
the gap between their levels with random signs over the rows (|T| is about 2 Eh, the closest levels of
24 waters 3e-5 Eh apart, of 100 waters 3e-6, of 300 waters 5e-7, those closer than 1e-7 |T| are
orthogonalised): 1e-14 up to 24 waters, 1e-13 at 100, 1e-12 at 300.  The products by L and L^-T add
N^1/2 eps cond(S)^1/2, about 3e-14 and 1e-13.  So 1e-13, 1e-12 and 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702


def _defect(calc, z, x):
    r = calc.calculate_flat([0, len(z)], z, x, compute_gradient=False)
    assert r.status[0] == 0
    mats = calc.molecule_matrices(0)
    occ = mats["occupations"]
    assert (np.minimum(np.abs(occ), np.abs(occ - 2.0)) == 0.0).all()
    P, S = mats["P"], mats["S"]
    return np.abs(P @ S @ P - 2.0 * P).max()


@pytest.mark.parametrize("waters, tolerance", [(1, 1e-13), (3, 1e-13), (8, 1e-13), (12, 1e-13), (16, 1e-13), (24, 1e-13),
                                                (64, 1e-12), (96, 1e-12), (100, 1e-12), (300, 1e-11)])
def test_density_is_idempotent(waters, tolerance):
    from gfn1_rs import BatchCalculator, workloads
    z, x = workloads.water_cluster(waters, 1)
    calc = BatchCalculator(electronic_temperature=0.0, energy_tolerance=1e-8, charge_tolerance=1e-6)
    assert _defect(calc, np.asarray(z, dtype=np.uint8), x * A2B) <= tolerance


# Dipoles (e bohr) of converged clusters from two pivoted inverse iterations a vector, 11 SCC iterations.
PIVOTED = {
    64: (-5.0507841532555195, -2.5011513752365238, -2.242295170734069),
    96: (-1.0689928934077546, 5.421291680811105, -4.97470914740497),
    300: (-9.431410176973088, -0.3492062994294059, -8.125087326047243),
}


@pytest.mark.parametrize("waters, tolerance", [(64, 1e-12), (96, 2e-12), (300, 2e-11)])
def test_dipole_is_that_of_two_pivoted_solves(waters, tolerance):
    """The charges take the overlap of the orbitals and the SCC's response multiplies it by about ten, so
    two sets of vectors as orthogonal as above (1e-13, 1e-13, 1e-12) agree in the dipole to ten times that."""
    from gfn1_rs import BatchCalculator, workloads
    z, x = workloads.water_cluster(waters, 1)
    r = BatchCalculator(energy_tolerance=1e-8, charge_tolerance=1e-7).calculate_flat([0, len(z)], z, x * A2B)
    want = np.array(PIVOTED[waters])
    assert r.status[0] == 0 and r.iterations[0] == 11
    assert np.abs(r.dipole[0] - want).max() <= tolerance * np.linalg.norm(want)
