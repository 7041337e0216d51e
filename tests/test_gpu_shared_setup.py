"""Setup and gradient with one CTA per molecule (a batch that fills the GPU)
against several CTAs and eight lanes per pair (a molecule on its own): one
launch for up to 16 atoms, several beyond, with and without d shells and
halogen-bond donors.

Tolerance: both evaluate the same sums in another order (1e-15 relative of terms
of at most 1 Eh), which the tight SCC amplifies by at most about 1e4: 1e-10 Eh,
1e-9 Eh/bohr, 1e-9 e."""
import numpy as np
import pytest

from conftest import smoke_molecule

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702
TIGHT = dict(energy_tolerance=1e-10, charge_tolerance=1e-8)


def _molecules(fixtures):
    from gfn1_rs import workloads
    out = [(np.array([2]), np.zeros((1, 3)))]
    for n in (1, 5, 6):  # 3, 15 and 18 atoms: either side of the one-launch limit
        z, x = workloads.water_cluster(n, 40 + n)
        out.append((z, x * A2B))
    z, x = out[2]
    out.append((np.append(z, 2), np.vstack([x, [[25.0, 0, 0]]])))                 # 16 atoms
    out.append((np.append(z, [2, 2]), np.vstack([x, [[25.0, 0, 0], [0, 25.0, 0]]])))  # 17
    out += [smoke_molecule(fixtures, n) for n in ("phosphine", "ferrocene")]
    rec = fixtures["halogen_tests"]["CH3Br...OH2 halogen bond"]
    out.append((np.array(rec["numbers"]), np.array(rec["positions_angstrom"]) * A2B))
    rng = np.random.default_rng(5)
    far = [np.array(rec["positions_angstrom"]) * A2B + 40.0 * k + rng.normal(0, 0.02, (len(rec["numbers"]), 3))
           for k in range(2)]
    out.append((np.array(rec["numbers"] * 2), np.vstack(far)))  # more than 16 atoms with donors
    return out


def test_single_molecules_equal_the_full_batch(gpu_calc, fixtures):
    from gfn1_rs import BatchCalculator
    mols = _molecules(fixtures)
    assert {len(z) for z, _ in mols} >= {1, 3, 15, 16, 17, 18}
    calc = BatchCalculator(**TIGHT)
    copies = 4 * 148 // len(mols) + 1  # at least four CTAs for each SM
    allm = mols * copies
    off = np.concatenate([[0], np.cumsum([len(z) for z, _ in allm])]).astype(np.int32)
    full = calc.calculate_flat(off, np.concatenate([z for z, _ in allm]), np.concatenate([x for _, x in allm]))
    assert np.all(full.status == 0)
    for m, (z, x) in enumerate(mols):
        r = calc.calculate_flat([0, len(z)], z, x)
        assert r.status[0] == 0 and r.iterations[0] == full.iterations[m]
        assert np.abs(r.terms[0] - full.terms[m]).max() <= 1e-10
        assert np.abs(r.gradient - full.gradient[off[m]:off[m + 1]]).max() <= 1e-9
        s0, s1 = full.shell_offsets[m], full.shell_offsets[m + 1]
        assert np.abs(r.shell_charges - full.shell_charges[s0:s1]).max() <= 1e-9
