"""Reductions of large molecules that a thread-block cluster or a grid holds on chip,
at the sizes where the class changes (8 CTAs up to 384 AOs, 16 up to 768, the SMs of
the GPU above, the blocked reduction of the first columns above 2368) and where slot
rows and columns fill up.

Tolerance: both reductions are backward stable, so the eigenvalues of F' agree to
about N eps |F'| (1e-12 Eh at 769 AOs) and a converged SCC of the same iterations
amplifies that by at most about 1e4 (the charge response over the smallest orbital
gaps): 1e-7 Eh, 1e-7 Eh/bohr and 1e-7 e hold with a margin; against the oracle, which
converges to 1e-10 Eh and 1e-8 e, the same."""
import os

import numpy as np
import pytest

from test_gpu_scc_sizes import TIGHT, molecule

pytestmark = pytest.mark.gpu

SIZES = (193, 255, 257, 320, 383, 384, 385, 513, 767, 768, 769)


def _calculate(mols, panel):
    from gfn1_rs import BatchCalculator
    old = os.environ.pop("GFN1_WIDE_PANEL", None)
    if panel:
        os.environ["GFN1_WIDE_PANEL"] = panel
    try:
        off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
        return off, BatchCalculator(**TIGHT).calculate_flat(off, np.concatenate([z for z, _ in mols]),
                                                            np.concatenate([x for _, x in mols]))
    finally:
        os.environ.pop("GFN1_WIDE_PANEL", None)
        if old is not None:
            os.environ["GFN1_WIDE_PANEL"] = old


def spread(nao):
    """Water clusters of 24 and one of the rest 40 A apart, so that the gap does not
    close with size, and helium atoms for the remainder."""
    z, x = [], []
    left, k = nao, 0
    while left:
        zz, xx = molecule(min(left, 192))
        z.append(zz)
        x.append(xx + np.array([75.0 * (k % 4), 75.0 * (k // 4), 1.3 * k]))
        left -= min(left, 192)
        k += 1
    return np.concatenate(z), np.concatenate(x)


@pytest.mark.parametrize("sizes", [(777,), (1183, 1001, 801), (2368,), (2369,), (2401, 300)])
def test_grid_and_blocked_reductions_agree(sizes):
    """One molecule on all SMs, several that share them, and more rows than they hold."""
    mols = [spread(n) for n in sizes]
    _, r = _calculate(mols, None)
    _, b = _calculate(mols, "16")
    assert (r.status == 0).all() and (b.status == 0).all()
    assert np.array_equal(r.iterations, b.iterations)
    assert np.abs(r.energy - b.energy).max() <= 1e-7
    assert np.abs(r.gradient - b.gradient).max() <= 1e-7
    assert np.abs(r.shell_charges - b.shell_charges).max() <= 1e-7


@pytest.mark.parametrize("sizes", [SIZES, (384,) * 17, (768, 320, 769)])
def test_cluster_and_blocked_reductions_agree(oracle_mod, sizes):
    mols = [molecule(n) for n in sizes]
    off, r = _calculate(mols, None)
    _, b = _calculate(mols, "16")
    assert (r.status == 0).all() and (b.status == 0).all()
    assert np.array_equal(r.iterations, b.iterations)
    assert np.abs(r.energy - b.energy).max() <= 1e-7
    assert np.abs(r.gradient - b.gradient).max() <= 1e-7
    assert np.abs(r.shell_charges - b.shell_charges).max() <= 1e-7
    for m, n in enumerate(sizes):
        if sizes is SIZES and n in (193, 385):
            o = oracle_mod.run(*mols[m], options=oracle_mod.make_options(**TIGHT))
            assert r.iterations[m] == o.iterations and abs(r.energy[m] - o.energy) <= 1e-7
            assert np.abs(r.gradient[off[m]:off[m + 1]] - o.gradient).max() <= 1e-7


@pytest.mark.parametrize("copies, distance", [(25, 90.0), (25, 16.0)])
def test_degenerate_and_close_eigenvalues(oracle_mod, copies, distance):
    """Copies of one water on a lattice: orbitals degenerate to rounding far apart
    (inverse iteration in a cluster), split by 1e-9 to 1e-4 Eh closer (twisted
    factorisation, then orthogonalised chains).  Energies are invariant under the
    mixing of degenerate orbitals, so the tolerance is the one above."""
    z1, x1 = molecule(8)
    at = np.array([[i % 3, (i // 3) % 3, i // 9] for i in range(copies)], dtype=float) * distance
    z = np.tile(z1, copies)
    x = (x1[None, :, :] + at[:, None, :]).reshape(-1, 3)
    _, r = _calculate([(z, x)], None)
    o = oracle_mod.run(z, x, options=oracle_mod.make_options(**TIGHT))
    assert r.status[0] == 0 and r.iterations[0] == o.iterations
    assert abs(r.energy[0] - o.energy) <= 1e-7
    assert np.abs(r.gradient - o.gradient).max() <= 1e-7
    assert np.abs(r.shell_charges - o.shell_charges).max() <= 1e-7


def test_back_transformation_beyond_shared_memory():
    """At 2920 AOs the columns of the back-transformation stay in global memory, at 2880
    in shared memory; the difference here is 40 helium atoms too far away to interact."""
    z, x = spread(2880)
    he = np.array([[-200.0 - 60.0 * k, 40.0, 10.0] for k in range(40)])
    more = (np.concatenate([z, np.full(40, 2, np.uint8)]), np.concatenate([x, he]))
    _, r = _calculate([(z, x), more, (np.array([2], np.uint8), np.zeros((1, 3)))], None)
    assert (r.status == 0).all() and r.iterations[0] == r.iterations[1]
    assert abs(r.energy[1] - r.energy[0] - 40 * r.energy[2]) <= 1e-7
    n = len(z)
    assert np.abs(r.gradient[n:2 * n] - r.gradient[:n]).max() <= 1e-7
