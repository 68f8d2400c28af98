"""Atom readouts around the sizes at which they change their way out: one piece of the pinned block (21,845
atoms), several, the whole block (174,762 atoms) and the device buffer beyond it. Same bytes as where
pinned memory is refused and all go through the device buffer."""

import subprocess

import numpy as np
import pytest

from test_gpu_readout import FAKE, _read

pytestmark = pytest.mark.gpu


# 21,845 and 21,846 atoms; 107,995; 174,762 and 174,763
@pytest.mark.parametrize("cells", [[((18, 17, 18), 187), ((18, 17, 18), 186)], [((30, 30, 30), 5)],
                                   [((36, 36, 34), 1494)], [((36, 36, 34), 1493)]])
def test_same_bytes_by_either_way(tmp_path, cells):
    src, lib = tmp_path / "fake.c", str(tmp_path / "fake.so")
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", lib, str(src), "-ldl"], check=True)
    want, got = _read(tmp_path, "refused", cells, lib), _read(tmp_path, "pinned", cells, None)
    for k in want.files:
        assert np.array_equal(want[k], got[k]), k
    import md_driver_module as m
    assert np.array_equal(got[f"start_{len(cells) - 1}_{m.ATOM_POSITIONS}"], got["positions_in"])
