"""The argument behind the CRT reconstruction's one-rounding path (CPU).

`crt_round` in eigen_b200/csrc/crt.cu splits the exact remainder R (|R| <= P/2) at fixed places into
A = floor(R / 2^kA), the 52 bits B below and, for kB = kA - 52 > 0, the bits below those, which set
B's last bit when any is nonzero: A 2^52 + B is R / 2^kB rounded to odd, and one rounding of it to
nearest is that of R while it is at least 2^55.  Restated here with exact Python integers for every
modulus count and checked against the exactly rounded value on random remainders, ties and lone sticky
bits, both signs, and at the ends of the range."""
from __future__ import annotations

import math
import random

import pytest

from _helpers import DBL_MIN, crt_model, exact_rn, remainders


def one_path(R: int, escale: int, bits: int):
    """crt_round past its range fix; None where it takes the magnitude path."""
    kL = bits + 1
    kA = kL - 51 if kL > 103 else 52
    kB = kA - 52
    A = R >> kA  # floor
    assert abs(A) <= 1 << 51 and 0 <= kB < 32
    B = (R >> kB) & ((1 << 52) - 1)
    if R & ((1 << kB) - 1):
        B |= 1
    d = float(A * 2 ** 52 + B)  # one rounding of exact operands, as the FMA
    if abs(d) < (2.0 ** 56 if kB else 1.0):
        return None
    try:
        v = math.ldexp(d, kB + escale)
    except OverflowError:
        return None
    if v == 0.0 or abs(v) < DBL_MIN or math.isinf(v):
        return None
    return v


@pytest.mark.parametrize("moduli", range(8, 17))
def test_one_path_rounds_like_exact_rounding(moduli):
    P = crt_model().modulus_product(moduli)
    half = P // 2
    bits = half.bit_length()
    rng = random.Random(moduli)
    ends = [s * (half - d) for s in (1, -1) for d in range(3)]
    kept = 0
    for R in [*remainders(bits, rng, 8000), *ends]:
        if abs(R) > half:
            continue
        escale = rng.choice([0, -60, -120, -900, -1000 - rng.randrange(80), 800 + rng.randrange(150)])
        got = one_path(R, escale, bits)
        if got is not None:
            assert got == exact_rn(R, escale), (R, escale)
            kept += 1
    assert kept > 1000
