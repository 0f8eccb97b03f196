"""The exact Riemann solver's shared-divisor quotients (Divisor, csrc/riemann.cuh)
are the correctly rounded ones: equal to IEEE division bit for bit."""
import ctypes as C

import numpy as np
import pytest

from m2c_b200 import abi


def mantissas(rng, n, kind):
    """Numbers in [1, 2): random, within a few units of 1 or of 2, or short."""
    if kind == "random":
        return 1.0 + rng.random(n)
    if kind == "short":
        return 1.0 + rng.integers(0, 2 ** 20, n) / 2.0 ** 20
    k = rng.integers(0, 64, n) * 2.0 ** -52
    return 1.0 + k if kind == "low" else 2.0 - 2.0 ** -52 - k


@pytest.mark.parametrize("ka", ["random", "low", "high", "short"])
@pytest.mark.parametrize("kb", ["random", "low", "high", "short"])
def test_quotients_are_correctly_rounded(host_riemann_lib, ka, kb):
    rng = np.random.default_rng(11)
    n = 200000
    # the range mid_range admits, with its ends
    a = mantissas(rng, n, ka) * 2.0 ** rng.integers(-400, 400, n) * rng.choice([-1.0, 1.0], n)
    b = mantissas(rng, n, kb) * 2.0 ** rng.integers(-400, 400, n)
    q = np.empty(n)
    host_riemann_lib.host_divisor.argtypes = [C.c_int] + [C.POINTER(C.c_double)] * 3
    host_riemann_lib.host_divisor(n, abi.dptr(a), abi.dptr(b), abi.dptr(q))
    assert np.array_equal(q, a / b)
