"""The node table of the overlap areas (csrc/bg3_area.cuh) against its formula, and what area_segment
says of its differences: {sqrt(1 - s s), asin(s)} at s = i / 128, each as two floats."""
import os
import re
import struct
from decimal import Decimal, getcontext

import numpy as np

from braingrid_gb300 import build as bgbuild

getcontext().prec = 60


def nodes():
    with open(os.path.join(bgbuild.CSRC, "bg3_area.cuh")) as f:
        body = re.search(r"area_nodes\[92\] = \{(.*?)\n\};", f.read(), re.S).group(1)
    rows = re.findall(r"\{([^{}]*)\}", body)
    return [[float.fromhex(v.strip().rstrip("f")) for v in r.split(",")] for r in rows]


def f32(v):
    return struct.unpack("f", struct.pack("f", v))[0]


def asin(x):
    """The Taylor series, which 60 digits end."""
    term, total, k = x, x, 0
    while abs(term) > Decimal(10) ** -55:
        k += 1
        term = term * x * x * (2 * k - 1) / (2 * k)
        total += term / (2 * k + 1)
    return total


def test_nodes_are_their_formula():
    table = nodes()
    assert len(table) == 92
    for i, (ch, cl, ah, al) in enumerate(table):
        s = Decimal(i) / 128
        for hi, lo, exact in ((ch, cl, (1 - s * s).sqrt()), (ah, al, asin(s))):
            assert hi == f32(float(exact)) and lo == f32(float(exact - Decimal(hi)))
            assert abs(Decimal(hi) + Decimal(lo) - exact) <= Decimal(2) ** -50


def test_products_differ_exactly():
    """m c - M t of an angle and its nearest node: the two rounded products lie within a factor of
    two, so that their difference is exact, but for the 256 sines from 1 / 256 on at the first node,
    where both are multiples of the difference's last place."""
    table = nodes()
    for i in range(1, 92):
        t = i / 128.0
        for m in ((i - 0.5) / 128 * (1 + 2.0 ** -15 if i == 1 else 1), (i + 0.5) / 128):
            p1, p2 = m * table[i][0], (1 - m * m) ** 0.5 * t
            assert 0.5 < p1 / p2 < 2.0, i
    c, t = np.float32(table[1][0]), np.float32(1 / 128)
    m = (np.float32(2.0 ** -8) * (1 + np.arange(512) * 2.0 ** -23)).astype(np.float32)
    big = np.sqrt(1 - m.astype(np.float64) ** 2).astype(np.float32)
    for M in (big, np.nextafter(big, np.float32(0)), np.nextafter(big, np.float32(2))):
        p1, p2 = m * c, M * t
        assert np.array_equal((p1 - p2).astype(np.float64), p1.astype(np.float64) - p2.astype(np.float64))
