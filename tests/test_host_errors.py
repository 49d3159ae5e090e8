"""Host code around launches, on a CUDA runtime without a device
(tests/fake_cudart.c): what is refused before memory is taken or a kernel
runs, and what becomes of a launch that fails.  No GPU is used: each test is a
child process with the stand-in preloaded, in which kernels do nothing.
"""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), "/usr/local/cuda")

PRELUDE = r"""
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import horsepower_gb300
from horsepower_gb300.abi import V0, H_B, H_C, H_E, H_I, H_L
import numpy as np
fake = C.CDLL(None)
L = horsepower_gb300.load(build_if_missing=False)
fake.cudaMalloc.argtypes = [C.c_void_p, C.c_size_t]

def column(typ, n, width):
    p = C.c_void_p()
    assert fake.cudaMalloc(C.byref(p), n * width) == 0
    v = V0()
    v.typ, v.len, v.g = typ, n, p.value
    return v

def count(*names):
    return [fake.fake_count(k.encode()) for k in names]

up, down = (L.vec(np.array([a]), H_B) for a in (True, False))
"""


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    if not os.path.exists(os.path.join(ROOT, "horsepower_gb300", "libhgpu.so")):
        pytest.skip("libhgpu.so is not built")
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    r = subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-w", "-I" + os.path.join(CUDA, "include"), "-o", so,
                        os.path.join(HERE, "fake_cudart.c")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(body, **env):
        r = subprocess.run([sys.executable, "-c", PRELUDE + body, ROOT], capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so, **env))
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_rows_beyond_the_row_ids(child):
    """@order and @group by radix passes refuse more than 2^32 rows, whose row
    ids do not fit 32 bits, before a pass runs; 2^32 rows, one more than the
    counted passes' positions hold, take the look-back passes.  (The stand-in's
    key statistics read as if every bit varied.)"""
    child(r"""
one, two = (lambda x: x), (lambda x: L.list([x, x]))
for n, rc, passes in ((2**32 - 1, 0, "k_rx_scatter"), (2**32, 0, "k_onesweep"), (2**32 + 1, 99, None)):
    for typ, width, shape in ((H_I, 4, one), (H_L, 8, one), (H_I, 4, two)):
        x = shape(column(typ, n, width))
        dirs = [L.vec(np.array([a] * (2 if shape is two else 1)), H_B) for a in (True, False)]
        for call in (lambda: L.rc("pfnOrderBy", x, dirs[0]), lambda: L.rc("pfnOrderBy", x, dirs[1]), lambda: L.rc("pfnGroup", x)):
            fake.fake_reset()
            L.lib.setHeapOffset(0)
            assert call() == rc, (n, typ, L.lib.hgpuLastError())
            ran = [k for k in ("k_rx_scatter", "k_onesweep") if count(k)[0]]
            assert ran == ([passes] if passes else []), (n, typ, ran)
x = column(H_C, 2**32 + 1, 1)
assert L.rc("pfnOrderBy", x, up) == 99 and L.rc("pfnGroup", x) == 99
""")


@pytest.mark.parametrize("kernel,err,rc,passes", [
    ("", 0, 100, True),                # nothing fails: the stand-in's barrier result reads as one that gave up
    ("k_qs_depths", 720, 0, True),     # cudaErrorCooperativeLaunchTooLarge: the depths take launches of their own
    ("k_qs_depths", 801, 0, True),     # cudaErrorNotSupported: the same
    ("k_qs_depths", 1, 100, False),    # any other refusal is the call's error
    ("k_qs_depths", 719, 100, False),
    ("k_qs_ranges", 1, 100, False),    # a failed launch before it is not taken for its refusal
])
def test_quicksort_launch_errors(child, kernel, err, rc, passes):
    """The quicksort's resident kernel may be refused, which has a path of its
    own; every other failed launch of the sort is reported."""
    child(r"""
kernel, err, rc, passes = %r, %d, %d, %r
x = column(H_E, 10_000, 8)
fake.fake_reset()
if kernel:
    fake.fake_fail(kernel.encode(), err)
fake.fake_poke(b"k_qs_whole", 1, 32, 4, 1)  # QsCounters::nbig: one range for the depths
got = L.rc("pfnOrderBy", x, up)
assert got == rc, (got, L.lib.hgpuLastError())
took, own = count("k_qs_depths", "k_qs_count")
if not kernel:
    assert took == 1 and b"barrier" in L.lib.hgpuLastError()
else:
    assert took == 0 and (own > 0) == passes, own
""" % (kernel, err, rc, passes))


def test_quicksort_scratch(child):
    """A quicksort of n rows takes less than 60 bytes of scratch a row: its two
    buffers hold the elements of the ranges listed on the way as well."""
    child(r"""
n = 4_000_000
x = column(H_E, n, 8)
fake.fake_reset()
fake.fake_poke(b"k_qs_whole", 1, 32, 4, 1)  # QsCounters::nbig: one range for the depths
assert L.rc("pfnOrderBy", x, up) == 0, L.lib.hgpuLastError()
assert count("k_qs_move")[0] > 0
""", HGPU_SCRATCH_LIMIT_MB=str(4_000_000 * 60 >> 20))


def test_group_trie_columns(child):
    """@group_trie reads its second column over the first one's length: a list
    without one, or with a shorter one, and a plain vector are refused before
    anything is read."""
    child(r"""
a, b, c = (column(H_C, n, 1) for n in (5000, 4999, 5000))
# (a node behind the one-column list, which a reader of two columns would take)
one = L.list([a, c]); one.len = 1
for x, rc in ((one, 1), (L.list([]), 1), (a, 1), (L.list([a, b]), 5), (L.list([a, c]), 0), (L.list([b, a]), 0)):
    fake.fake_reset()
    assert L.rc("pfnGroupTrie", x) == rc, (x.len, L.lib.hgpuLastError())
    assert (count("k_trie_present")[0] > 0) == (rc == 0)
""")


@pytest.mark.parametrize("cols,kernel,arg,row", [(1, "k_qs_whole", 1, 53), (2, "k_qs_mode", 8, 68)])
def test_quicksort_scratch_of_listed_ranges(child, cols, kernel, arg, row):
    """The lists of ranges and the trades add little to what the quicksort's
    buffers take: 52 bytes of scratch a row for a vector, 67 for a list of
    columns."""
    child(r"""
n, cols, row = 4_000_000, %d, %d
x = column(H_E, n, 8)
fake.fake_reset()
fake.fake_poke(%r, %d, 32, 4, 1)  # QsCounters::nbig: one range for the depths
assert L.rc("pfnOrderBy", *((x, up) if cols == 1 else (L.list([x] * cols), L.vec(np.array([True] * cols), H_B)))) == 0
assert count("k_qs_move")[0] > 0
""" % (cols, row, kernel.encode(), arg), HGPU_SCRATCH_LIMIT_MB=str(4_000_000 * row >> 20))


def test_radix_scratch_of_small_orders(child):
    """The digit counts of a radix pass are sized by its chunks: an order of
    20,000 rows takes less than a megabyte of scratch."""
    child(r"""
for typ, width in ((H_I, 4), (H_L, 8)):
    x = column(typ, 20_000, width)
    for d in (up, down):
        fake.fake_reset()
        assert L.rc("pfnOrderBy", x, d) == 0, L.lib.hgpuLastError()
        assert count("k_rx_scatter")[0] > 0
""", HGPU_SCRATCH_LIMIT_MB="1")
