"""The grid teams' sums (csrc/resident.cuh, team_sum_fixed) in exact integer arithmetic: a
block's partial becomes two words of 40 bits, scaled by an earlier sum's exponent, and a sum
that is too small beside that earlier one is repeated another way.  Just above that line,
with every block's truncation at its worst, the sum must still hold 52 bits."""
import os
import re
from fractions import Fraction

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dav-qed2d_b200", "csrc", "resident.cuh")


def test_sum_keeps_52_bits_at_the_line():
    src = open(SRC).read()
    scale = int(re.search(r"\(1023 \+ (\d+) - ex\) << 52\);   // exact", src).group(1))
    line = int(re.search(r"s >= __longlong_as_double\(\(long long\)\(1023 - (\d+) \+ ex\) << 52\)", src).group(1))
    blocks, ex = 148, 0
    total = Fraction(1, 1 << line) * (1 << ex)
    # partials whose remainder beyond the low word is as large as it gets
    unit = Fraction(1, 1 << (scale + 40 - ex))
    partial = (total / blocks // unit + Fraction(9999, 10000)) * unit
    words = 0
    for _ in range(blocks):
        y = partial * (1 << scale) / (1 << ex)
        hi = y.numerator // y.denominator
        lo = int((y - hi) * (1 << 40))
        words += (hi << 40) + lo
    got = Fraction(words, 1 << 40) / (1 << scale) * (1 << ex)
    want = blocks * partial
    assert abs(got - want) < want / (1 << 52)
