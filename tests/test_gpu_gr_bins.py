"""g(r)'s FP32 bin estimate with its FP64 recheck: bit for bit the oracle's histograms on cells
without a potential file, for bins from coarse to finer than the estimate resolves (every pair
then takes the FP64 test), pairs placed on bin edges (undisplaced lattice), tile remainders, one
to three types, and histograms beyond the shared-memory limit."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, oracle

pytestmark = pytest.mark.gpu

METHODS = ["calculate_pair_correlation", "calculate_pair_correlations",
           "calculate_partial_pair_correlation"]


@pytest.mark.parametrize("types,edges,vacancies,n_rg,sigma", [
    (1, (4, 4, 4), 0, 2, 0.08), (2, (5, 4, 6), 3, 700, 0.08), (2, (5, 5, 5), 0, 500, 0.0),
    (3, (6, 7, 6), 5, 3000, 0.08), (2, (8, 8, 8), 1, 9000, 0.08), (2, (4, 4, 4), 2, 300000, 0.08)])
def test_gr_bitwise(types, edges, vacancies, n_rg, sigma):
    c = generic_case(generic_tables(types), edges, vacancies, sigma_ang=sigma)
    half = 0.5 * c.box.diagonal().min()
    drg = half / n_rg
    c.rg = [(k + 0.5) * drg for k in range(n_rg)]
    d, o = gpu(c), oracle(c)
    for mode in range(3):
        getattr(d, METHODS[mode])()
        g_o, gp_o = o.pair_correlation(mode)
        if mode != 2:
            assert g_o.sum() > 0 and np.array_equal(np.array(d.gr), g_o)
        if mode != 0:
            assert gp_o.sum() > 0 and np.array_equal(np.array(d.gr_partial), gp_o)
