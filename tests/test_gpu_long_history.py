"""Charge mixing with long histories (more than 16 vectors are eliminated by the whole CTA, eight entries of a
row at a time where a row has them), and after fewer requested iterations than the ladder's last rung has.

Tolerances that nothing meets keep the mixing at work after convergence, through every rung of the ladder; the
last one, at 3000 K, then ends at the oracle's converged charges for that temperature.  Tolerance: its steps
move the charges by rounding, 1e-15 e amplified by the solve's conditioning (weights of 1e5 over a
regularisation of 1e-2, at most 1e7), and the oracle converges to 1e-9 e: 1e-8 e, and 1e-9 Eh in the energy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702


@pytest.mark.parametrize("history, max_scc, dense_n", [(15, 250, None), (16, 250, None), (17, 250, None), (18, 250, None),
                                                       (33, 30, None), (112, 250, None), (130, 3, None), (145, 250, None),
                                                       (250, 2, None), (17, 250, "4"), (130, 3, "4")])
def test_long_histories_match_the_oracle(oracle_mod, monkeypatch, history, max_scc, dense_n):
    from gfn1_rs import BatchCalculator, workloads
    if dense_n:  # the large-molecule path
        monkeypatch.setenv("GFN1_DENSE_N", dense_n)
    opts = dict(energy_tolerance=1e-300, charge_tolerance=1e-300, max_scc=max_scc, scc_broyden_size=history)
    mols = [workloads.water_cluster(n, 60 + n) for n in (1, 2, 5)]
    off = np.concatenate([[0], np.cumsum([len(z) for z, _ in mols])]).astype(np.int32)
    z, x = np.concatenate([z for z, _ in mols]).astype(np.uint8), np.concatenate([x for _, x in mols]) * A2B
    r = BatchCalculator(**opts).calculate_flat(off, z, x)
    assert (r.status != 0).all() and (r.iterations == 250).all()
    for m in range(len(mols)):
        a, b, s0, s1 = off[m], off[m + 1], r.shell_offsets[m], r.shell_offsets[m + 1]
        o = oracle_mod.run(z[a:b], x[a:b], gradient=False, options=oracle_mod.make_options(
            energy_tolerance=1e-11, charge_tolerance=1e-9, electronic_temperature=3000.0))
        assert np.abs(r.shell_charges[s0:s1] - o.shell_charges).max() <= 1e-8
        assert abs(r.energy[m] - o.energy) <= 1e-9
