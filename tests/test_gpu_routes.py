"""Rules that choose between kernels: which kernels a call launches on either
side of a rule's line, and that its result is the same on both.

Bar: bit-exact.
"""
import ctypes as C

import numpy as np
import pytest

from horsepower_gb300.abi import DTYPE, H_E, H_F, H_H, H_I, H_L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import horsepower_gb300
    L = horsepower_gb300.load()
    L.lib.hgpuProfileRead.argtypes = [C.c_int32, C.POINTER(C.c_char_p), C.POINTER(C.c_double), C.POINTER(C.c_longlong)]
    return L


def launches(L, fn):
    """fn()'s result and its launches by kernel name."""
    L.lib.hgpuProfileReset()
    L.lib.hgpuProfile(1)
    try:
        out = fn()
    finally:
        L.lib.hgpuProfile(0)
    names, ms, n = (C.c_char_p * 256)(), (C.c_double * 256)(), (C.c_longlong * 256)()
    k = L.lib.hgpuProfileRead(256, names, ms, n)
    got = {names[i].decode(): n[i] for i in range(k)}
    L.lib.hgpuProfileReset()
    return out, got


@pytest.mark.parametrize("n", [3, 255, 257, 2048 + 5, 70_001])
@pytest.mark.parametrize("typ,span,kernel", [(H_I, 4000, "member"), (H_H, 30_000, "member"), (H_L, 60_000, "member"),
                                             (H_I, 2 ** 31 - 1, "member_hash"), (H_L, 2 ** 62, "member_hash"),
                                             (H_F, 0, "member_hash"), (H_E, 0, "member_hash")])
def test_member_routes(gpu, typ, span, kernel, n):
    """@member looks eight keys up at a time in a direct table and one at a
    time in a hashed one, where eight take the registers that hide the walk."""
    rng = np.random.default_rng(n + typ)
    if span:
        x, other = (rng.integers(-span // 2, span // 2, m).astype(DTYPE[typ]) for m in (1000, n))
        x[:2] = [-(span // 2), span // 2 - 1]
    else:
        x, other = (rng.standard_normal(m).astype(DTYPE[typ]) for m in (1000, n))
        other[::7] = np.nan
    y = np.where(rng.random(n) < 0.5, rng.choice(x, n), other)
    z, got = launches(gpu, lambda: gpu.call("pfnMember", gpu.vec(y, typ), gpu.vec(x, typ)))
    assert np.array_equal(gpu.to_py(z), np.isin(y, x))
    assert {k for k in got if k.startswith("member")} == {kernel}, got
    gpu.free_inputs()
