"""Device functions of the particle kernel on their own (tests/device/checks.cu, built beside the library): the pair
arithmetic gives the floats of the GPU's IEEE operations, and the bounded wait tests its phase before it gives up."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'device', 'libchecks.so')
WAIT_TIMEOUT = 1                # ST_WAIT_TIMEOUT


@pytest.fixture(scope='module')
def checks():
    assert os.path.exists(PATH), 'built by make -C zpic-parallel_b200'
    return ctypes.CDLL(PATH)


def bits(x):
    return int(np.float32(x).view(np.uint32))


QLIM = 2.0 ** 96                # the pair operations' range ends below


def test_roots_and_reciprocals(checks):
    """Every float of [1, 2^96)."""
    bad = (ctypes.c_ulonglong * 2)(1, 1)
    assert checks.check_roots(ctypes.c_uint32(bits(1.0)), ctypes.c_uint32(bits(QLIM)), bad) == 0
    assert list(bad) == [0, 0]


def test_energy_terms(checks):
    """utsq / ( sqrt( 1 + utsq ) + 1 ) for every float of [0, 2^96), denormals included: the divisor is 2 where the
    remainder of the quotient is not a normal number."""
    bad = (ctypes.c_ulonglong * 1)(1)
    assert checks.check_energy_terms(ctypes.c_uint32(0), ctypes.c_uint32(bits(QLIM)), bad) == 0
    assert bad[0] == 0


def test_quotients(checks):
    """Every significand of the divisor, exponents of [0, 48), 64 numerators each."""
    bad = (ctypes.c_ulonglong * 1)(1)
    assert checks.check_quotients(64, bad) == 0
    assert bad[0] == 0


@pytest.mark.parametrize('arrive,limit', [(1, 1), (1, 100), (0, 1), (0, 2), (0, 200)])
def test_bounded_wait(checks, arrive, limit):
    out = (ctypes.c_int * 3)()
    assert checks.check_wait(arrive, limit, out) == 0
    assert out[0] == arrive
    assert out[2] == (0 if arrive else WAIT_TIMEOUT)
