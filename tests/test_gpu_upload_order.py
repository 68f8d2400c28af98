"""What a driver uploads between launches (block maps of a launch shape, cell grids, replica states,
list offsets) is in place before the kernels that read it, whatever else keeps the device's legacy
stream busy: the same bits as on a quiet device. A driver's stream does not wait for the legacy one."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, gpu_atoms
from test_gpu_mlp_reset import _BusyLegacyStream

pytestmark = pytest.mark.gpu


def _results(c):
    out = []
    d = gpu(c)
    for tpa, blocks in ((8, 148 * 8), (4, 148 * 32), (16, 148 * 2), (1, 148 * 64)):
        d.set_launch(tpa, tpa, blocks, blocks)
        d.run(7, 3, 1)
        point, neighbors = d.neighbor_list()
        out += [np.array(point), np.array(neighbors), gpu_atoms(d, "forces"),
                np.array(d.born_elasticity_tensor)]
    return out


# all pairs, and cells (3,430 atoms)
@pytest.mark.parametrize("rcut,edges,vacancies", [(4.5, (5, 5, 5), 3), (5.0, (9, 9, 11), 134)])
def test_same_bits_beside_a_busy_legacy_stream(rcut, edges, vacancies):
    c = generic_case(generic_tables(2, rcut=rcut), edges, vacancies, ensemble=2, T=600.0)
    want = _results(c)
    with _BusyLegacyStream():
        for _ in range(2):
            for got, ref in zip(_results(c), want):
                assert np.array_equal(got, ref)
