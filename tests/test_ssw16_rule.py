"""The rule that sends SSW tasks to the packed 16-bit kernel: for every set of penalties, the
longest read it admits keeps the kernel's scaled 16-bit numbers from wrapping.  Scores are
scaled by 32, their low five bits hold a row.  Every read up to the longest is taken, so the
longest one's numbers are the largest."""
import ctypes as C

import numpy as np

import strobealign_gb300 as sa


class Scores(C.Structure):
    _fields_ = [(n, C.c_uint8) for n in ("match", "mismatch", "gap_open", "gap_extend")] + [("end_bonus", C.c_uint32)]


def _max_qlen():
    f = sa.lib()["_ZN2sa14ssw16_max_qlenERKNS_11AlignScoresE"]  # sa::ssw16_max_qlen(const AlignScores&)
    f.argtypes, f.restype = [C.POINTER(Scores)], C.c_uint32
    return lambda *s: f(C.byref(Scores(*s, 10)))


def test_no_number_wraps():
    longest = _max_qlen()
    admitted = 0
    for match in range(1, 256):
        for extend in range(256):
            # the opening penalty only decides whether the scores are taken at all
            q = longest(match, 8, 255, extend) if extend < 255 else 0
            for opening in {min(255, extend + 1), min(255, extend + 12)}:
                assert longest(match, 8, opening, extend) == (q if opening > extend else 0)
            if not q:
                continue
            admitted += 1
            # the best score with its row
            assert 32 * match * q + 31 <= np.iinfo(np.int16).max, (match, extend, q)
            # word mode: the lazy-F raise loses a gap extension for every row of a lane, in
            # two pieces, from 0 on
            assert -32 * extend * (-(-q // 8)) >= np.iinfo(np.int16).min, (match, extend, q)
    assert admitted > 100
    assert longest(2, 8, 12, 1) == 511 and longest(3, 8, 12, 1) == 340  # as long as the others allow
    assert longest(0, 8, 12, 1) == 0 and longest(2, 8, 12, 12) == 0 and longest(2, 65, 12, 1) == 0
