"""The lengths that the FFT passes hold with compile-time indices are those of the rule that
the table states, no more and no fewer (reads the source)."""

import math
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _table():
    src = open(os.path.join(ROOT, "pyfourier_b200", "csrc", "pfb_fft.cuh")).read()
    pairs = []
    for name in ("PFB_FFT_TWO", "PFB_FFT_TWO_BIG"):
        body = re.search(rf"#define {name}\(X\)((?:.*\\\n)*.*)", src).group(1)
        pairs.append([(int(a), int(b)) for a, b in re.findall(r"X\((\d+), (\d+)\)", body)])
    return pairs


def _plan(n):
    """stage_plan's two stages of n: radices to 16, the least sum, else the first to 32 and the
    more even split; None when it takes others."""
    two = [(a, n // a) for a in range(16, 1, -1) if n % a == 0 and 2 <= n // a <= a]
    if two:
        return min(two, key=sum)
    big = [(a, n // a) for a in range(17, 33) if n % a == 0 and 8 <= n // a <= a]
    return big[0] if big else None


def test_table_is_the_rule():
    small, big = _table()
    extents = [n for n in range(64, 257) if n % 16 == 0 or n % 20 == 0]
    lengths = {math.ceil(n * f) for n in extents for f in (1, 1.25, 1.5, 2)}
    want = {_plan(n) for n in lengths if n >= 80 and _plan(n)}
    assert sorted(small + big) == sorted(want)
    assert all(a <= 16 for a, _ in small) and all(a > 16 for a, _ in big)
