"""The polynomial that takes a quarter of the portion attention's exponentials (heads of 64), restated in float32 with the
coefficients that stand in the kernel: as close to 2^x as the special-function unit's ex2, and zero where that is."""

import re
from pathlib import Path

import numpy as np

SOURCE = Path(__file__).resolve().parent.parent / "tokasaurus_b200" / "csrc" / "attention_tc.cu"


def poly(x):
    body = SOURCE.read_text().split("void exp2_poly(")[1].split("\n}")[0]
    lowest = np.float32(re.search(r"fmaxf\(x0, (-[0-9.]+)f\)", body).group(1))
    coefficients = [np.float32(c) for c in re.findall(r"twice\(([0-9.]+)f\)", body)]
    assert lowest == -127 and len(coefficients) == 6 and coefficients[-1] == 1
    shift = np.float32(12582912.0)
    x = np.maximum(x.astype(np.float32), lowest)
    t = x + shift
    f = x - (t - shift)
    p = np.full_like(f, coefficients[0])
    for c in coefficients[1:]:  # a product and a sum of float32 are rounded once (float64 holds the product whole)
        p = (p.astype(np.float64) * f + np.float64(c)).astype(np.float32)
    return (p.view(np.int32) + np.left_shift(t.view(np.int32), 23)).view(np.float32)


def test_polynomial_is_as_close_as_ex2():
    x = np.linspace(-125.9, 20, 4_000_001).astype(np.float32)
    want = np.exp2(x.astype(np.float64))
    # the fit's own 9.2e-8, a rounding of each of the last two steps (2^-25 each where the result is near one, 2^-24 below it)
    assert (np.abs(poly(x) - want) / want).max() < 2.0e-7


def test_ends_of_the_range():
    x = np.linspace(-127, -126, 1001).astype(np.float32)
    assert (np.abs(poly(x) - np.exp2(x.astype(np.float64))) <= 2.0 ** -126).all() and (poly(x) >= 0).all()
    assert (poly(np.asarray([-127.0, -127.5, -150.0, -1e30, -np.inf], dtype=np.float32)) == 0).all()
