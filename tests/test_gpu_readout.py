"""Atom readouts where pinned host memory is refused (a fake cudaHostAlloc in a child process returns
cudaErrorMemoryAllocation once the drivers are made): the same bytes as with it, for small replicas and
for one whose fields take several pieces of the driver's readout block."""

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdio.h>
static int refuse;
void fake_refuse(int on) { refuse = on; }
int cudaHostAlloc(void **p, size_t bytes, unsigned flags) {
    if (refuse) {
        fprintf(stderr, "REFUSED\n");
        return 2;
    }
    void *rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    int (*real)(void **, size_t, unsigned) = (int (*)(void **, size_t, unsigned))dlsym(rt, "cudaHostAlloc");
    return real(p, bytes, flags);
}
"""

CHILD = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests", {root!r} + "/mdelast_b200/lib"]
import numpy as np
import md_driver_module as m
from generic import generic_case, generic_tables
from test_gpu_list_paths import _batch
t = generic_tables(1, rcut=4.5)
cases = [generic_case(t, e, v, seed=k) for k, (e, v) in enumerate({cells!r})]
b = _batch(cases)
if {refuse!r}:
    import ctypes
    ctypes.CDLL(None).fake_refuse(1)
out = {{}}
for when in ("start", "stepped"):
    for r in range(len(cases)):
        for f in range(m.ATOM_POSITIONS, m.ATOM_EKIN + 1):
            out[f"{{when}}_{{r}}_{{f}}"] = np.array(b.atoms(r, f))
    b.run(2, 20, 1, False)
out["positions_in"] = np.asarray(cases[-1].positions)
np.savez({path!r}, **out)
"""


def _read(tmp_path, name, cells, preload):
    path = str(tmp_path / (name + ".npz"))
    env = dict(os.environ)
    if preload:
        env["LD_PRELOAD"] = preload
    code = CHILD.format(root=ROOT, cells=cells, path=path, refuse=bool(preload))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert ("REFUSED" in p.stderr) == bool(preload)
    return np.load(path)


# 500 and 1,001 atoms; 186,624 atoms, 4.5 MB a vector field
@pytest.mark.parametrize("cells", [[((5, 5, 5), 0), ((6, 6, 7), 7)], [((36, 36, 36), 0)]])
def test_pinned_memory_refused(tmp_path, cells):
    src, lib = tmp_path / "fake.c", str(tmp_path / "fake.so")
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", lib, str(src), "-ldl"], check=True)
    want, got = _read(tmp_path, "pinned", cells, None), _read(tmp_path, "refused", cells, lib)
    assert set(want.files) == set(got.files)
    for k in want.files:
        assert np.array_equal(want[k], got[k]), k
    last = len(cells) - 1
    import md_driver_module as m
    assert np.array_equal(want[f"start_{last}_{m.ATOM_POSITIONS}"], want["positions_in"])
