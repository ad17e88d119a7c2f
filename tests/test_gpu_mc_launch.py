"""Packet counts at which the transport's launch changes: one lane per warp, the first count that
takes two, a full grid and one more than it. Tallies of a run split in two by packet ranges add up to
those of the whole run (FP64 sums in another order: 1e-12 of the largest)."""
import numpy as np
import pytest

from mcmatlab_b200 import configs, mexargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 4736, 4737, 151552, 151553])
def test_split_runs_add_up(n):
    from mcmatlab_b200 import native
    mc_in = mexargs.prepare_mc(configs.standard_tissue_cube(n=20, nPhotons=n, seed=n))
    whole = native.mc_run(mc_in, tallies=True)["tallies"]
    a = n // 3 + 1
    first = native.mc_run(dict(mc_in, nPhotonsRequested=float(a)), tallies=True)["tallies"]
    rest = native.mc_run(dict(mc_in, nPhotonsRequested=float(n - a), packetOffset=a), tallies=True)["tallies"]
    assert whole[-2] == n  # launched packets
    assert np.max(np.abs(first + rest - whole)) <= 1e-12 * np.max(np.abs(whole))
