"""The Fermi level against the oracle's.  With an open gap at 300 K every level inside the gap gives the same
occupations, so the electron count fixes it only by its rounding, some 37 kT above the HOMO: it is the oracle's
(and the reference's) only where the levels are counted in the same order.

Tolerance: the bisection ends at adjacent numbers and the eigenvalues agree to the SCC's convergence (1e-8 e,
at most 1e-8 Eh): 1e-7 Eh.  A count in another order is off by 1e-4 Eh and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702
TIGHT = dict(energy_tolerance=1e-10, charge_tolerance=1e-8)


def test_fermi_level_of_gapped_molecules(oracle_mod):
    from gfn1_rs import BatchCalculator, workloads
    mols = [workloads.water_cluster(n, 30 + n) for n in (1, 2, 3, 5, 8, 9, 12, 13, 16, 20, 24, 25, 32, 40)]
    off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
    z, x = np.concatenate([z for z, _ in mols]).astype(np.uint8), np.concatenate([x for _, x in mols]) * A2B
    r = BatchCalculator(**TIGHT).calculate_flat(off, z, x, compute_gradient=False)
    for m in range(len(mols)):
        o = oracle_mod.run(z[off[m]:off[m + 1]], x[off[m]:off[m + 1]], gradient=False,
                           options=oracle_mod.make_options(**TIGHT))
        assert r.status[m] == 0 and r.iterations[m] == o.iterations
        assert abs(r.fermi_level[m] - o.fermi_level) <= 1e-7
