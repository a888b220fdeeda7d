"""CPU: the polynomial that takes an eighth of the attention's exponentials (``ex2_poly2`` in csrc/attention.cu), evaluated
with its own coefficients in float32 as the kernel does (Horner with fused multiply-adds), against 2^f over its range.

Bound: the fit's own error, 9.4e-8, plus half a unit in the last place of every partial sum, carried through the steps
behind it: 1.6e-7 in all.  2^f at f = 0 is 1 exactly."""
import os
import re

import numpy as np

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed-xfold_b200", "csrc", "attention.cu")


def test_exp2_polynomial_over_its_range():
    with open(SOURCE) as f:
        src = f.read()
    at = src.index("float2 ex2_poly2(float2 y)")
    body = src[at:src.index("\n}\n", at)]
    coef = [np.float32(v) for v in re.findall(r"make_float2\(([\d.]+)f, \1f\)", body)]
    assert len(coef) == 6
    f = np.linspace(-0.5, 0.5, 1_000_001).astype(np.float32)
    fma = lambda a, b, c: (a.astype(np.float64) * b.astype(np.float64) + np.float64(c)).astype(np.float32)
    q, rounding = np.full_like(f, coef[0]), np.zeros(f.shape)
    for c in coef[1:]:
        q = fma(q, f, c)
        rounding = rounding * np.abs(f) + 0.5 * np.spacing(np.abs(q))
    want = np.exp2(f.astype(np.float64))
    bound = 9.4e-8 + (rounding / want).max()
    assert bound < 1.65e-7
    assert np.abs(q / want - 1).max() < bound
    assert q[f == 0][0] == 1
