"""A source shape whose kernel gave up a bounded wait is an error, not a result: both entry points (laph_sourceshape,
laph_solver_sourceshape) return what laph_sourceshape_status makes of the flag the kernel leaves beside psi."""
import pytest

import laph_eigsys_b200 as lb
from laph_eigsys_b200 import _lib


def test_no_flag_is_success():
    assert lb.lib.laph_sourceshape_status(0) == _lib.LAPH_OK


@pytest.mark.parametrize("flag", [1, -1])
def test_a_wait_that_gave_up_is_an_error(flag):
    assert lb.lib.laph_sourceshape_status(flag) == _lib.LAPH_ECUDA
    with pytest.raises(lb.LaphError) as e:
        lb.check(lb.lib.laph_sourceshape_status(flag), "laph_sourceshape")
    assert e.value.status == _lib.LAPH_ECUDA and "not valid" in str(e.value)
