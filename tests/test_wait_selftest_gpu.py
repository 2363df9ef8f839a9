"""The bounded-wait self-test covers every wait of the Gauss-Seidel kernels:
rows of other CTAs and of the own CTA in the tile kernel, and the row-by-row
kernel of 25 x 25 and 27 x 27 blocks -- three launches, each ended by its time
limit."""
import ctypes as C

import pytest

import mgldg

pytestmark = pytest.mark.gpu


def test_every_wait_runs_out(ctx):
    before = ctx.prof()["gauss_seidel"][0]
    st = C.c_int(-1)
    assert mgldg.lib().mgldg_selftest_wait_timeout(ctx.h, 2_000_000, C.byref(st)) == mgldg.OK
    assert ctx.prof()["gauss_seidel"][0] - before == 3
    assert st.value == mgldg.ERR_TIMEOUT
