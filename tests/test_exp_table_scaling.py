"""The FP64 kernels' exp puts 2^m into the exponent field of the table value before
its last FMA (csrc/common.cuh, exp_tab).  Emulated exactly on the host: within 1.5 ulp
down to the least normal number and within 1.5 units of 2^-1074 below it, the same bits
as a multiplication by 2^m afterwards while the result is normal."""

import math
import re
import struct
from fractions import Fraction

import numpy as np

from test_exp_table import _const, _exp_tab, _fma, _header, _table


def _kernel(s, tab, inv_l, l_hi, l_lo):
    t = _fma(s, inv_l, 6755399441055744.0)
    kd = t - 6755399441055744.0
    k = struct.unpack("<q", struct.pack("<d", t))[0] & 0xFFFFFFFF
    k -= (k >> 31) << 32
    r = _fma(-kd, l_lo, _fma(-kd, l_hi, s))
    q = _fma(_fma(_fma(r, 1.0 / 120.0, 1.0 / 24.0), r, 1.0 / 6.0), r, 0.5)
    p = _fma(r * r, q, r)
    m = max(-1022, min(1023, k >> 6))
    bits = struct.unpack("<Q", struct.pack("<d", tab[k & 63]))[0]
    tj = struct.unpack("<d", struct.pack("<Q", bits + (m << 52)))[0]
    return float("inf") if Fraction(tj) * (1 + Fraction(p)) >= 2 ** 1024 else _fma(tj, p, tj)


def test_the_header_has_this_form():
    body = re.search(r"double exp_tab\(.*?\n\}", _header(), re.S).group(0)
    assert re.search(r"__hiloint2double\(__double2hiint\(t0\) \+ \(m << 20\), __double2loint\(t0\)\);\s*"
                     r"return fma\(tj, p, tj\);", body)


def test_error_and_bits():
    tab = _table()
    consts = (_const("kInvL"), _const("kLhi"), _const("kLlo"))
    rng = np.random.default_rng(1)
    least = math.log(2.0 ** -1022)
    for s in np.concatenate([rng.uniform(-80, 80, 800), rng.uniform(-708, 709, 800)]):
        s = float(s)
        got, ref = _kernel(s, tab, *consts), math.exp(s)
        assert abs(got - ref) <= 1.5 * math.ulp(ref), s
        assert got == _exp_tab(s, tab, *consts)
    for s in least + rng.uniform(-0.005, 0.005, 200):  # around the least normal number
        s = float(s)
        got, ref = _kernel(s, tab, *consts), math.exp(s)
        assert abs(got - ref) <= 1.5 * max(math.ulp(ref), 2.0 ** -1074), s
    assert _kernel(0.0, tab, *consts) == 1.0
