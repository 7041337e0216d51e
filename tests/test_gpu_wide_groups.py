"""Large molecules in groups that share the workspace slots one after the other (what bounds the memory
of a large batch): the same results, bit for bit, as with every molecule in a slot of its own, since up
to 768 AOs a molecule's arithmetic does not depend on the others that run beside it; with a fallback ladder in one
group and rejected molecules among them."""
import os

import numpy as np
import pytest

from test_gpu_scc_sizes import molecule

pytestmark = pytest.mark.gpu


def _run(mols, slot_mb, options):
    from gfn1_rs import BatchCalculator
    old = os.environ.pop("GFN1_WIDE_SLOT_MB", None)
    if slot_mb:
        os.environ["GFN1_WIDE_SLOT_MB"] = str(slot_mb)
    try:
        off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
        calc = BatchCalculator(**options)
        z, x = np.concatenate([m[0] for m in mols]), np.concatenate([m[1] for m in mols])
        rs = [calc.calculate_flat(off, z, x) for _ in range(2)]  # the second one reuses the layout
        return rs[0], rs[1], [calc.molecule_matrices(m) for m in (0, len(mols) - 1)]
    finally:
        os.environ.pop("GFN1_WIDE_SLOT_MB", None)
        if old is not None:
            os.environ["GFN1_WIDE_SLOT_MB"] = old


@pytest.mark.parametrize("slot_mb", [1, 12])
@pytest.mark.parametrize("options", [dict(energy_tolerance=1e-8, charge_tolerance=1e-6), dict(max_scc=6)])
def test_groups_do_not_change_results(slot_mb, options):
    """1 MB: a group per molecule; 12 MB: two or three of the smaller ones together."""
    sizes = (193, 200, 255, 320, 201, 385, 193)
    mols = [molecule(n) for n in sizes]
    mols.insert(2, (np.array([2], np.uint8), np.zeros((1, 3))))  # one on the one-SM path
    a = _run(mols, None, options)
    b = _run(mols, slot_mb, options)
    for r in (a[1], b[0], b[1]):
        for name in ("energy", "gradient", "shell_charges", "dipole", "iterations", "status", "rung"):
            assert np.array_equal(getattr(a[0], name), getattr(r, name)), name
    for u, v in zip(a[2], b[2]):
        assert np.array_equal(u["P"], v["P"]) and np.array_equal(u["fock"], v["fock"])
