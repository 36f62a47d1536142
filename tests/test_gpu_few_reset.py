"""Few-sample runs on device buffers before and after the device's context is reset (with
every handle gone): the scratch pool of the first context is not used in the second."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes as C, gc, sys
import numpy as np
from mc_dagprop_gb300 import batching, workloads as W
from mcd_testlib import lib

cu = C.CDLL("libcuda.so.1")
flat = W.layered_dag_fast(np.random.default_rng(1), 40, 4, 3, [1, 2], 1800.0)
n, ones = 5, []
for k in range(2):
    prop = batching.compile_dag(flat, list(W.GEN_TWO_TYPES))
    E = prop.node_count()
    d = C.c_uint64()
    assert cu.cuMemAlloc_v2(C.byref(d), C.c_size_t(8 * (E + 1) * n)) == 0
    seeds, out = np.arange(n, dtype=np.int64), np.empty((E, n))
    assert cu.cuMemcpyHtoD_v2(d, seeds.ctypes.data_as(C.c_void_p), C.c_size_t(8 * n)) == 0
    assert lib().mcd_run_device(C.c_void_p(prop._handle()), d.value, n, d.value + 8 * n, None, None, n, None) == 0
    assert lib().mcd_dag_check(C.c_void_p(prop._handle())) == 0
    assert cu.cuMemcpyDtoH_v2(out.ctypes.data_as(C.c_void_p), C.c_uint64(d.value + 8 * n), C.c_size_t(8 * E * n)) == 0
    ones.append(out.copy())
    assert cu.cuMemFree_v2(d) == 0
    del prop
    gc.collect()
    if k == 0:
        assert cu.cuDevicePrimaryCtxReset_v2(0) == 0
assert np.array_equal(*ones)
print("same rows")
"""


def test_runs_on_both_sides_of_a_reset(cuda):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same rows" in r.stdout, r.stdout + r.stderr
