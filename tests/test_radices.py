"""Radix schedules of the azimuth lengths: a compiled schedule wherever one has the length, by whichever radices
it was compiled, and otherwise two or three near factors, for every length that a split can give.
"""
from __future__ import annotations

import ctypes as C
import re

import pytest

import build as B


def _radices(lib, n, strided):
    out = (C.c_int * 16)()
    k = lib.asarf_emu_radices(n, int(strided), out)
    return list(out[:k])


@pytest.mark.parametrize("strided,macro,most", [(True, "ASARF_STRIDED_SCHEDULES", 9), (False, "ASARF_BLOCK_SCHEDULES", 8)])
def test_compiled_schedules_first(emu_lib, strided, macro, most):
    compiled = {}
    for v in B._cases("params.h", macro):
        r = [int(x) for x in v.split(", ")]
        compiled[r[0] * r[1] * r[2]] = r
    assert len(compiled) == len(B._cases("params.h", macro))  # one schedule a length
    for n in range(4, 641):
        m = n
        for q in (2, 3, 5, 7):
            while m % q == 0:
                m //= q
        if m != 1:
            continue
        r = _radices(emu_lib, n, strided)
        prod = 1
        for x in r:
            prod *= x
        assert prod == n and all(2 <= x <= most for x in r), (n, r)
        if n in compiled:
            assert r == compiled[n]
        elif any(n % a == 0 and n // a <= most for a in range(2, most + 1)) and n > most:
            assert len(r) == 2 and r[0] >= r[1]
    # the planner names no length of its own
    text = (B.CSRC / "host.cpp").read_text()
    body = text[text.index("std::vector<int> strided_radices"):text.index("static int largest_divisor_to_root")]
    assert not re.search(r"n == [0-9]", body)
