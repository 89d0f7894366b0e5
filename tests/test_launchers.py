"""The wrappers through which the bindings call the kernels' launchers, and the same through ctypes."""

import ctypes

import pytest
import torch

from lalamo_b200 import native


@pytest.fixture(scope="module")
def both():
    if native.library_path() is None:
        pytest.skip("the kernel library is not built")
    return native.launchers(), native._CtypesLaunchers(native.library())


def test_every_launcher_has_a_wrapper(both):
    for name in native._prototypes():
        assert callable(getattr(both[0], name)) and callable(getattr(both[1], name))


def test_arguments(both):
    for calls in both:
        assert calls.lb_recurrent_value_floats(9, 1) == 2 * 64 * 8
        assert calls.lb_recurrent_pack_floats(ctypes.c_int(3), 5, 0) == 3 * 5 + 3
        # no tokens: nothing is launched, and nothing is read through the addresses
        assert calls.lb_add_bias(torch.zeros(4), None, 0, 4, 0, None) == 0
    assert both[0].lb_recurrent_value_floats(torch.tensor(9), True) == 2 * 64 * 8
    with pytest.raises(TypeError):
        both[0].lb_recurrent_value_floats(9)
    with pytest.raises((TypeError, AttributeError)):
        both[0].lb_recurrent_value_floats("9", 1)
