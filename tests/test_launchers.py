"""The wrappers through which the bindings call the kernels' launchers, and the same through ctypes."""

import ctypes
import re
from pathlib import Path

import numpy as np
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


def test_every_launcher_that_the_bindings_call(both):
    """The bindings' own names, and what the sources define by another look at them than the wrappers' (any result type, anywhere on a line)."""
    package = Path(native.__file__).parent
    called = set(re.findall(r"\blb_\w+", (package / "ops.py").read_text()))
    defined = {name for path in native.source_files() for name in re.findall(r"\b(lb_\w+)\s*\([^;{}]*\)\s*\{", re.sub(r"//[^\n]*", "", path.read_text()))}
    assert called and called <= defined
    # for programs without torch, which call it through ctypes
    without = {"lb_attention_decode_static"}
    for name in (called | defined) - without:
        assert callable(getattr(both[0], name)) and callable(getattr(both[1], name)), name


INTEGERS = [(9, 1024), (True, 512), (np.int64(9), 1024), (np.array(9), 1024), (torch.tensor(9), 1024), (ctypes.c_int(9), 1024), (ctypes.c_longlong(9), 1024), (2 ** 32 + 9, 1024), (2 ** 70 + 9, 1024)]


@pytest.mark.parametrize("given,result", INTEGERS)
def test_what_is_a_number(both, given, result):
    """What ``ctypes.c_int`` takes, and ctypes' own objects."""
    for calls in both:
        assert calls.lb_recurrent_value_floats(given, 1) == result


@pytest.mark.parametrize("given", [None, 9.0, np.float32(9), "9", torch.tensor(9.0), torch.zeros(2, dtype=torch.int32), ctypes.c_float(9), ctypes.c_void_p(None), [9]])
def test_what_is_none(both, given):
    for calls in both:
        with pytest.raises(TypeError):
            calls.lb_recurrent_value_floats(given, 1)


@pytest.mark.parametrize("given", [1, 1.5, True, np.float32(1.5), np.int64(2), np.array(1.5), torch.tensor(1.5), torch.tensor(2), ctypes.c_float(1.5)])
def test_what_is_a_real_number(both, given):
    """What ``ctypes.c_float`` takes (a scaling of no elements: nothing is launched)."""
    for calls in both:
        assert calls.lb_scale(None, given, 0, None, 0.0) == 0


@pytest.mark.parametrize("given,error", [(None, TypeError), ("1", TypeError), (10 ** 400, OverflowError), ([1.0], TypeError)])
def test_what_is_no_real_number(both, given, error):
    for calls in both:
        with pytest.raises(error):
            calls.lb_scale(None, given, 0, None, 0.0)


@pytest.mark.parametrize("given", [None, 0, torch.zeros(1), ctypes.c_void_p(None), ctypes.c_void_p(64)])
def test_what_is_an_address(both, given):
    for calls in both:
        assert calls.lb_scale(given, 1.0, 0, None, 0.0) == 0


def test_the_number_of_arguments(both):
    for calls in both:
        for arguments in ((9,), (9, 1, 1)):
            with pytest.raises(TypeError):
                calls.lb_recurrent_value_floats(*arguments)
