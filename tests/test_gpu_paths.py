"""Edges of the kernels that a rule on sizes, types or alignment selects:
each path against the oracle, or against the general path over the same data.

Bar: bit-exact (integers, permutations, and f64 sums against the oracle's
restatement of the fixed summation order).
"""
import ctypes as C
import os

import numpy as np
import pytest

from horsepower_gb300.abi import Builtins, H_B, H_C, H_E, H_I, H_L  # noqa: F401

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def libs():
    import subprocess
    import horsepower_gb300
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle"), "port"], check=True)
    ora = Builtins(os.path.join(ROOT, "oracle", "_build", "liboracle.so"), "oracle")
    ora.lib.hgoTreeSumF64.restype = C.c_double
    ora.lib.hgoTreeSumF64.argtypes = [C.c_void_p, C.c_longlong]
    return horsepower_gb300.load(), ora


@pytest.mark.parametrize("sizes", [
    [33, 64, 255, 256, 257, 288, 511, 512],            # a block of segments one warp takes each
    [513, 514, 767, 768, 769, 1024, 4095, 4096],       # a block of segments all warps share
    [33, 513, 34, 4096, 512, 40, 2049, 256, 700] * 9,  # both in one block, and a last block not full
])
def test_mid_size_groups(libs, sizes):
    """Groups of 33 to 4096 rows: sums equal the fixed tile tree of their rows
    bit for bit, min and max equal numpy's, on either side of 512 rows."""
    gpu, ora = libs
    rng = np.random.default_rng(len(sizes))
    key = np.repeat(np.arange(len(sizes), dtype=np.int64) + 70_000 * (np.arange(len(sizes)) % 2), sizes)
    rng.shuffle(key)
    pay = rng.standard_normal(key.size) * 10.0 ** rng.integers(-8, 8, key.size)
    ipay = rng.integers(-2 ** 31, 2 ** 31, key.size).astype(np.int32)
    g = gpu.call("pfnGroup", gpu.vec(key, H_L))
    vals = gpu.call("pfnValues", g)
    keys = gpu.to_py(gpu.call("pfnKeys", g))
    sums = gpu.to_py(gpu.call("hgpuGroupSum", gpu.vec(pay, H_E), vals))
    lo = gpu.to_py(gpu.call("hgpuGroupMin", gpu.vec(ipay, H_I), vals))
    hi = gpu.to_py(gpu.call("hgpuGroupMax", gpu.vec(pay, H_E), vals))
    for gi, first in enumerate(keys):
        rows = np.flatnonzero(key == key[first])
        x = np.ascontiguousarray(pay[rows])
        want = ora.lib.hgoTreeSumF64(x.ctypes.data, x.size)
        assert sums[gi].tobytes() == np.float64(want).tobytes(), (len(rows), sums[gi], want)
        assert lo[gi] == ipay[rows].min() and hi[gi] == x.max()
    gpu.free_inputs()
