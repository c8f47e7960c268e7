"""Failing runtime calls, made on the host by a shim that answers one call of
the CUDA runtime with an error code: what the engine then reports and keeps.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
/* fail_memset(k): the k-th cudaMemsetAsync from now on returns
   cudaErrorInvalidValue without being performed */
static int left = 0;
void fail_memset(int k) { left = k; }
int cudaMemsetAsync(void *p, int v, size_t n, void *s) {
  static int (*real)(void *, int, size_t, void *) = 0;
  if (!real)  /* the runtime the engine has loaded */
    real = (int (*)(void *, int, size_t, void *))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMemsetAsync");
  if (left > 0 && --left == 0) return 1;
  return real(p, v, n, s);
}
/* fail_malloc(k, c): c cudaMalloc calls from the k-th from now on return
   cudaErrorMemoryAllocation without being performed */
static int skip = 0, fail = 0;
void fail_malloc(int k, int c) { skip = k - 1; fail = c; }
int cudaMalloc(void **p, size_t n) {
  static int (*real)(void **, size_t) = 0;
  if (!real)
    real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
  if (skip > 0) --skip;
  else if (fail > 0) { --fail; return 2; }
  return real(p, n);
}
"""

CHILD = r"""
import ctypes, sys
sys.path[:0] = [{root!r}, {pkg!r}]
import numpy as np
from pimc.engine import ChainParams, Engine, Mix, PimcError
shim = ctypes.CDLL({so!r})
def chains():
    e = Engine([ChainParams(dim=2, N=6, M=12, L=3.0, T=1.0, lam=0.5, harmonic_omega=1.0, seed=i) for i in range(3)],
               Mix(stage_slices=4, stage_max=4, swaps_per_sweep=6, swap_slices=4, swap_max=4, measure_every=1))
    e.set_launch(64, split_phases=1)
    return e
want = chains()
want.run_batched(2)
for k in (1, 2, 3):
    e = chains()
    shim.fail_memset(k)
    try:
        e.run_batched(2)
        failed = False
    except PimcError:
        failed = True
    shim.fail_memset(0)
    assert failed and e.stats(0).sweeps == 0, k
    e.run_batched(2)  # nothing of the failed capture is kept
    for c in range(3):
        st = e.stats(c)
        assert st.sweeps == 2 and st.measurements == 2, (k, st)
        np.testing.assert_array_equal(e.get_beads(c), want.get_beads(c))
    e.close()
print("child ok")
"""


CONTACT_CHILD = r"""
import ctypes, sys
sys.path[:0] = [{root!r}, {pkg!r}]
import numpy as np
from pimc.engine import ChainParams, Engine, Mix, PimcError, contact_table
shim = ctypes.CDLL({so!r})
tab = contact_table(1.16, 1.0 / 12, 4.0, 50)
def chain():
    return Engine(ChainParams(dim=2, N=20, M=12, L=3.0, T=1.0, lam=0.5, harmonic_omega=1.0, interactions=True,
                              r_a=1.0, semantics=1, seed=4),
                  Mix(stage_slices=4, stage_max=4, swaps_per_sweep=20, swap_slices=4, swap_max=4))
def attach(e, made):
    e.set_contact_propagator(1.16, 4.0, 50) if made else e.set_contact_table(tab, 4.0)
out = []
# all there; no room for the FP32 copy; (refused) no room at all, or for the
# quadrature's scratch, then asked again
for made, k, c in ((0, 1, 0), (1, 1, 0), (0, 1, 1), (1, 1, 1), (0, 1, 2), (1, 1, 2), (1, 2, 99)):
    e = chain()
    shim.fail_malloc(k, c)
    refused = c > 1
    try:
        attach(e, made)
        assert not refused, (made, k, c)
    except PimcError:
        assert refused, (made, k, c)
        assert e.contact_table()[0] is None
    shim.fail_malloc(1, 0)
    if refused:
        attach(e, made)
    e.run_batched(4)
    out.append((e.get_beads(), e.stats(0).accepts))
    e.close()
for x, a in out[1:]:
    np.testing.assert_array_equal(x, out[0][0])
    assert a == out[0][1]
print("child ok")
"""


def _child(code, tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    code = code.format(root=ROOT, pkg=os.path.join(ROOT, "pimc.jl_gb300"), so=str(so))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=240,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0 and "child ok" in r.stdout, r.stdout + r.stderr


def test_contact_tables_without_room(engine_lib, tmp_path):
    """a device without room for a table's FP32 copy decides from exact sums; one
    without room for the table or its quadrature refuses it, and takes it when
    asked again.  The chains are the same every way"""
    _child(CONTACT_CHILD, tmp_path)


def test_an_error_during_capture_is_reported_and_nothing_of_it_kept(engine_lib, tmp_path):
    """a launch step that fails while a sweep is captured: the call reports it,
    no sweep has run, and the next call sweeps as a new handle does"""
    _child(CHILD, tmp_path)
