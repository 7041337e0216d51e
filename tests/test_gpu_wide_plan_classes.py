"""Plans of the blocked reduction are kept per size class; sizes 2360 and 2400 AOs share one, but only
the larger has columns that do not fit on chip.  So the plan search runs for it although the smaller
came first, and not again."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A2B = 1.8897261246257702


def test_a_size_with_nothing_to_choose_does_not_settle_the_plan_of_one_with(capfd):
    from gfn1_rs import BatchCalculator, workloads
    saved = {k: os.environ.pop(k, None) for k in ("GFN1_WIDE_PANEL", "GFN1_WIDE_TIMING")}
    os.environ["GFN1_WIDE_TIMING"] = "1"
    try:
        z, x = workloads.water_cluster(300, 1)
        z, x = np.asarray(z, dtype=np.uint8), np.asarray(x) * A2B
        # the two sizes five at a time, a count that no other test uses for them
        counts = []
        for waters in (295, 300, 300):
            n = 3 * waters
            capfd.readouterr()
            r = BatchCalculator(energy_tolerance=1e-4, charge_tolerance=1e-3).calculate_flat(
                np.arange(6, dtype=np.int32) * n, np.tile(z[:n], 5), np.tile(x[:n], (5, 1)), compute_gradient=False)
            assert (r.status == 0).all()
            counts.append(capfd.readouterr().err.count("wide tune N"))
        assert counts[0] == 1 and counts[1] > 1 and counts[2] == 0
    finally:
        for k, v in saved.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v
