"""g(r) on bins finer than the FP32 estimate resolves, of a range that takes in few of the pairs or half
the box, with partial histograms that shared memory holds only at the cost of the occupancy, and
with total histograms beyond it for small and large cells: bit for bit the oracle's histograms; and fine
bins of a short range cost little more than coarse ones (the FP64 test of every pair: FP64 units instead
of FP32, no more)."""

import time

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, oracle

pytestmark = pytest.mark.gpu

METHODS = ["calculate_pair_correlation", "calculate_pair_correlations",
           "calculate_partial_pair_correlation"]


def _rg(c, rmax_ang, n_rg):
    half = 0.5 * c.box.diagonal().min()
    drg = (half if rmax_ang is None else rmax_ang * 1e-8) / n_rg
    return [(k + 0.5) * drg for k in range(n_rg)]


@pytest.mark.parametrize("types,edges,vacancies,rmax,n_rg", [
    (2, (5, 5, 5), 3, 3.0, 40000),     # fine, few pairs
    (2, (10, 11, 10), 5, 4.0, 12000),  # fine, few pairs, several tiles per block
    (1, (10, 11, 10), 1, None, 60000),  # fine, half the box
    (2, (12, 12, 12), 7, 6.0, 6000),   # partial: 72 KB for few pairs
    (3, (12, 11, 12), 2, None, 3000),  # partial: 72 KB for half the pairs
    (2, (5, 5, 5), 0, None, 30000),    # total beyond shared memory, small cell
    (2, (11, 11, 11), 2, None, 30000)])  # ... and a large one
def test_histograms_bitwise(types, edges, vacancies, rmax, n_rg):
    c = generic_case(generic_tables(types), edges, vacancies)
    c.rg = _rg(c, rmax, n_rg)
    d, o = gpu(c), oracle(c)
    for mode in range(3):
        getattr(d, METHODS[mode])()
        g_o, gp_o = o.pair_correlation(mode)
        if mode != 2:
            assert g_o.sum() > 0 and np.array_equal(np.array(d.gr), g_o)
        if mode != 0:
            assert gp_o.sum() > 0 and np.array_equal(np.array(d.gr_partial), gp_o)


def test_fine_bins_of_a_short_range():
    """32,000 atoms, range 6 A: bins of 0.0005 A against bins of 0.005 A. Queueing every pair of the cell,
    those out of range too, took 2.7 times as long."""
    ms = []
    for n_rg in (1200, 12000):
        c = generic_case(generic_tables(1), (20, 20, 20), 0)
        c.rg = _rg(c, 6.0, n_rg)
        d = gpu(c)
        t = []
        for _ in range(8):
            t0 = time.perf_counter()
            d.calculate_pair_correlation()
            d.gr
            t.append(time.perf_counter() - t0)
        ms.append(1e3 * min(t))
    assert ms[1] <= 1.8 * ms[0], ms
