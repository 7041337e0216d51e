"""Molecules beyond a cluster (769 AOs and more) are reduced by grids, a few at a time, or all together
by the blocked reduction, whichever their number and sizes make the faster: batches on both sides of that
rule, and one whose molecules leave it at different iterations, against the blocked reduction for all.

Tolerance: the two reductions' eigenvalues and vectors agree to N eps |F'| (1e-12 Eh at 1200 AOs, the
orbitals orthogonal to 1e-11), which a converged SCC of the same iterations amplifies by at most about a
hundred in these gapped clusters: 1e-9 Eh, Eh/bohr and e."""
import os

import numpy as np
import pytest

from test_gpu_cluster_reduction import spread

pytestmark = pytest.mark.gpu


def _run(mols, panel):
    from gfn1_rs import BatchCalculator
    old = os.environ.pop("GFN1_WIDE_PANEL", None)
    if panel:
        os.environ["GFN1_WIDE_PANEL"] = panel
    try:
        off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
        return BatchCalculator(energy_tolerance=1e-9, charge_tolerance=1e-7).calculate_flat(
            off, np.concatenate([z for z, _ in mols]), np.concatenate([x for _, x in mols]))
    finally:
        os.environ.pop("GFN1_WIDE_PANEL", None)
        if old is not None:
            os.environ["GFN1_WIDE_PANEL"] = old


@pytest.mark.parametrize("sizes", [(1200,) * 7, (1200,) * 9, (1400,) + (777,) * 12, (2400, 800, 800)])
def test_either_choice_agrees_with_the_blocked_reduction(sizes):
    rng = np.random.default_rng(len(sizes))
    mols = [(z, x + rng.normal(0.0, 0.02, x.shape)) for z, x in map(spread, sizes)]
    r, b = _run(mols, None), _run(mols, "16")
    assert (r.status == 0).all() and (b.status == 0).all()
    assert np.array_equal(r.iterations, b.iterations)
    assert np.abs(r.energy - b.energy).max() <= 1e-9
    assert np.abs(r.gradient - b.gradient).max() <= 1e-9
    assert np.abs(r.shell_charges - b.shell_charges).max() <= 1e-9
