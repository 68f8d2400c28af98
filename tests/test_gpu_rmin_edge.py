"""The r_min warning of the FP64 passes decides on the correctly rounded distance, as the oracle
does: a smallest distance at r_min itself, and one unit in the last place to either side of it. A
distance off by one unit warns where the oracle does not, or the other way round."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, oracle

pytestmark = pytest.mark.gpu


def _smallest(c):
    """The smallest distance [cm], in the operations of the oracle's minimum image."""
    L = c.box.diagonal()
    s = c.positions / L
    d = s[:, None] - s[None]
    d = (d - np.rint(d)) * L
    r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]
    np.fill_diagonal(r2, np.inf)
    return float(np.sqrt(r2.min()))


@pytest.mark.parametrize("neighbors", [True, False])
def test_distance_at_rmin(neighbors):
    seen = set()
    for seed in range(24):
        t = generic_tables(1, n_r=200, n_rho=200)
        c = generic_case(t, (4, 4, 4), 1, seed=seed, neighbors=neighbors)
        d = _smallest(c)
        for rmin in (np.nextafter(d, 0.0), d, np.nextafter(d, 1.0), np.nextafter(np.nextafter(d, 1.0), 1.0)):
            t.rmin_fatal = float(rmin)
            o = oracle(c).status()
            assert gpu(c).status == o, (seed, rmin - d)
            seen.add(o)
    assert len(seen) == 2  # both outcomes were met
