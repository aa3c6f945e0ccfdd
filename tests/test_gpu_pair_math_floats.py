"""The claims of csrc/pair_math.cuh for every float: roots as the walks (2^-60 to 2^60) and
the anisotropic pass (2^-96 to 1e30) take them, reciprocals of densities, and the quotients
by those roots whose reciprocal is not the rounded one, for all numerators of the smallest
binade that the host admits and of one in the middle."""
import ctypes as C

import pytest

from particles4all_b200 import _abi, _lib

pytestmark = pytest.mark.gpu


def counts(lo, hi, numerator):
    c = (C.c_uint64 * 4)()
    assert _lib.lib().p4a_test_pair_math(lo, hi, numerator, c) == 0
    return list(c)


@pytest.mark.parametrize("numerator", [2.0 ** -101, 1.0])
def test_walks(built, numerator):
    roots, recips, unrounded, quotients = counts(2.0 ** -60, 2.0 ** 60, numerator)
    assert roots == recips == quotients == 0
    assert 0 < unrounded < 60 * 64  # what the quotients were taken by


@pytest.mark.parametrize("lo,hi", [(2.0 ** -96, 2.0 ** -60), (2.0 ** 60, 2.0 ** 100)])
def test_roots_of_the_anisotropic_pass(built, lo, hi):
    assert counts(lo, hi, 1.0)[0] == 0


def test_bad_ranges(built):
    c = (C.c_uint64 * 4)()
    L = _lib.lib()
    for args in ((0.0, 1.0, 1.0), (1.0, 1.0, 1.0), (1.0, 2.0 ** 101, 1.0), (1.0, 2.0, 0.0), (1.0, 2.0, float("nan"))):
        assert L.p4a_test_pair_math(*args, c) == _abi.P4A_ERR_ARG
