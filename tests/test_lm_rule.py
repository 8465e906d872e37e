"""The LM kernel configuration (threads, slots) that the default rule names for every
direction count, luminance and RGB.  A pass is summed in threads / 32 - 1 parts, so the
choice is part of a fit's bits; the rule needs no GPU."""
import ctypes as C

import pytest

import tempestrenderer_b200 as svf

# first direction count of each run of equal choices, up to 160
LUM = {3: (128, 3), 60: (160, 3), 71: (128, 3), 72: (128, 2), 76: (160, 2), 90: (256, 2), 112: (160, 2),
       113: (256, 3), 131: (160, 3), 132: (256, 2)}
RGB = {3: (128, 3), 49: (160, 3), 58: (128, 2), 62: (160, 2), 73: (128, 2), 74: (256, 2), 92: (256, 3),
       108: (256, 2), 134: (256, 1)}


class _Choice(C.Structure):
    _fields_ = [("threads", C.c_int), ("slots", C.c_int), ("pairs", C.c_int)]


@pytest.mark.parametrize("rgb,want", [(False, LUM), (True, RGB)])
def test_default_choice_of_every_direction_count(rgb, want):
    rule = C.CDLL(svf.LIB_PATH)["_ZN3svf17lm_default_choiceEjmb"]   # svf::lm_default_choice
    rule.restype, rule.argtypes = _Choice, (C.c_uint32, C.c_uint64, C.c_bool)
    for n in range(3, 161):
        values = (3 if rgb else 1) * n * n
        c = rule(n, (values + 7) // 8 * 8, rgb)
        assert (c.threads, c.slots, c.pairs) == (*want[max(k for k in want if k <= n)], 0), n
