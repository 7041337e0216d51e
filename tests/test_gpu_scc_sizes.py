"""The persistent SCC kernel at the sizes where its tiling changes: matrices of
one row, one short of, equal to and one beyond a tile of 8, 32, 64, 96, 128 and
192 AOs (the last ones either side of the register-resident reductions and of
the large-molecule path), from water clusters and helium atoms (one AO each,
doubly occupied, so that small cases have every orbital occupied).

Tolerance: the device and the oracle take the same iterations (tight
convergence), so only rounding differs; the SCC amplifies the eigensolver's
few-ulp errors (1e-15 of |F| ~ 1 Eh) by at most about 1e4 (the charge response
over the smallest orbital gaps), so 1e-9 Eh, 1e-8 Eh/bohr and 1e-8 e hold with
a wide margin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702
TIGHT = dict(energy_tolerance=1e-10, charge_tolerance=1e-8)
SIZES = (1, 2, 3, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 192, 193)


def molecule(nao):
    from gfn1_rs import workloads
    nw, nhe = divmod(nao, 8)
    z, x = [], np.zeros((0, 3))
    if nw:
        zw, x = workloads.water_cluster(nw, 100 + nw)
        z = list(zw)
    r = 3.0 + np.abs(x).max(initial=0.0)
    he = np.array([[r + 2.1 * k, 0.3 * k, -0.2 * k] for k in range(nhe)]).reshape(-1, 3)
    return np.array(z + [2] * nhe, dtype=np.uint8), np.concatenate([x, he]) * A2B


def _check(r, m, z, x, o, off):
    a0, a1 = off[m], off[m + 1]
    s0, s1 = r.shell_offsets[m], r.shell_offsets[m + 1]
    assert r.status[m] == 0 and r.iterations[m] == o.iterations
    assert abs(r.energy[m] - o.energy) <= 1e-9
    assert np.abs(r.gradient[a0:a1] - o.gradient).max() <= 1e-8
    assert np.abs(r.shell_charges[s0:s1] - o.shell_charges).max() <= 1e-8


@pytest.mark.parametrize("copies", [1, 32])
def test_sizes_around_the_tiles(oracle_mod, copies):
    """One call with every size once (the wide CTAs of a small batch), and one
    with enough copies that the small sizes run on the narrow ones."""
    from gfn1_rs import BatchCalculator
    mols = [molecule(n) for n in SIZES]
    for n, (z, _) in zip(SIZES, mols):
        assert oracle_mod.sizes(z)[0] == n
    ref = [oracle_mod.run(z, x, options=oracle_mod.make_options(**TIGHT)) for z, x in mols]
    pick = [m for m in range(len(SIZES)) for _ in range(copies if SIZES[m] <= 65 else 1)]
    off = np.concatenate([[0], np.cumsum([len(mols[m][0]) for m in pick])]).astype(np.int32)
    r = BatchCalculator(**TIGHT).calculate_flat(off, np.concatenate([mols[m][0] for m in pick]),
                                                np.concatenate([mols[m][1] for m in pick]))
    small = sum(SIZES[m] <= 64 for m in pick)
    assert copies == 1 or small > 2 * 148  # more than the wide CTAs the GPU holds at once
    for i, m in enumerate(pick):
        _check(r, i, *mols[m], ref[m], off)
