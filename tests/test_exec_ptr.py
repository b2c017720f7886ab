"""Plan.exec_ptr takes device addresses as integers (or None, which the C ABI
refuses); objects that ctypes would pass by their host address are refused
before any call.  No GPU: the plan handle is null, so a call that is made
returns MCFFT_INVALID_PLAN."""
import ctypes

import pytest

import mcfft_b200 as mc


def _closed_plan():
    p = mc.Plan.__new__(mc.Plan)
    p._h = ctypes.c_void_p()
    return p


@pytest.mark.parametrize("bad", [b"host bytes", "text", (ctypes.c_float * 4)(), ctypes.c_char_p(b"x"),
                                 ctypes.c_void_p(4096), 4096.0])
@pytest.mark.parametrize("place", [0, 1, 3])
def test_exec_ptr_refuses_host_objects(place, bad):
    args = [4096, 8192, mc.FORWARD, 0]
    args[place] = bad
    with pytest.raises(TypeError):
        _closed_plan().exec_ptr(*args)


@pytest.mark.parametrize("args", [(4096, 8192), (None, 8192), (4096, 8192, mc.INVERSE, None), (True, 8192)])
def test_exec_ptr_passes_integers_on(args):
    with pytest.raises(mc.McfftError) as ei:
        _closed_plan().exec_ptr(*args)
    assert ei.value.code == mc.INVALID_PLAN
