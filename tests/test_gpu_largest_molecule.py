"""The largest molecule the engine takes: 1660 atoms, what the set-up kernel's 227 KB of shared memory
hold at 140 bytes an atom, whatever the elements.  One atom more is refused with a message that names
the size, and the other molecules of the call are not affected.

The molecules are helium droplets (random sites, every orbital filled, charges zero), so that their
energies add when they are far apart.  Tolerance: the sum of N levels and its rounding, N eps sum|f eps|
(1660 x 2e-16 x 3e3 Eh = 1e-9), times the growth over two diagonalisations: 1e-8 Eh and, for the gradient,
whose terms are local, 1e-9 Eh/bohr."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 1660


def droplet(n, seed):
    """n helium atoms on a jittered lattice of 5.5 bohr."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 5.5
    return np.full(n, 2, np.uint8), g + rng.uniform(-0.8, 0.8, g.shape)


def test_largest_molecule_and_one_atom_more():
    from gfn1_rs import BatchCalculator
    parts = [droplet(800, 1), droplet(LIMIT - 800, 2)]
    far = np.array([400.0, 0.0, 0.0])
    whole = (np.concatenate([parts[0][0], parts[1][0]]), np.concatenate([parts[0][1], parts[1][1] + far]))
    mols = parts + [whole]
    off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
    z, x = np.concatenate([m[0] for m in mols]), np.concatenate([m[1] for m in mols])
    calc = BatchCalculator()
    r = calc.calculate_flat(off, z, x)
    assert (r.status == 0).all()
    assert abs(r.energy[2] - r.energy[0] - r.energy[1]) <= 1e-8
    assert np.abs(r.gradient[LIMIT:] - r.gradient[:LIMIT]).max() <= 1e-9
    # one atom more, beside a molecule that is fine
    more = np.concatenate([whole[1], [[-30.0, 0.0, 0.0]]])
    off2 = np.array([0, 800, 800 + LIMIT + 1], np.int32)
    z2, x2 = np.full(off2[-1], 2, np.uint8), np.concatenate([parts[0][1], more])
    r2 = calc.calculate_flat(off2, z2, x2)
    assert r2.status[0] == 0 and r2.status[1] != 0
    assert abs(r2.energy[0] - r.energy[0]) <= 1e-8
    with pytest.raises(Exception, match=f"{LIMIT + 1} atoms.*{LIMIT}"):
        calc.calculate_flat(off2, z2, x2, raise_on_error=True)
