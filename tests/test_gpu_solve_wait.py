"""A one-launch triangular solve whose waits run out (its first block is never
solved) ends after the limit with an error that the host reads; the context and
the next solve are fine."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_wait_limit_is_reported(cuda, flame):
    expired = C.c_int(0)
    assert flame.lib().FLA_B200_solve_wait_check(C.byref(expired)) == flame.FLA_SUCCESS, flame.last_error()
    assert expired.value == 1
    assert flame.lib().FLA_B200_solve_wait_check(None) == flame.FLA_FAILURE
