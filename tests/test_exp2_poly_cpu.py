"""The polynomial that takes a share of the attention's exponentials (exp2_poly2): its coefficients are those of the fit that its comment
names, and the function with its fp32 roundings stays within the error that the comment states."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

STATED = 1.8e-7
F = np.float32


@pytest.fixture(scope="module")
def source():
    with open(os.path.join(ROOT, "eager-flash-attention_b200", "csrc", "fa_fwd_ws_sm100.cu")) as f:
        text = f.read()
    at = text.index("uint64_t exp2_poly2(")
    comment, body = text[text.rindex("}\n", 0, at):at], text[at:text.index("\n}\n", at)]
    coefficients = [float.fromhex(h) for h in re.findall(r"pack2\((0x1\.[0-9a-f]+p[-+]\d+)f, \1f\)", body)]
    assert len(coefficients) == 5                                # of f^5 to f; the constant term is 1
    return comment, coefficients


def test_coefficients_are_the_minimax_fit(source):
    """min over c of max |(1 + c1 f + ... + c5 f^5) / 2^f - 1| on [-1/2, 1/2], as a linear program over Chebyshev nodes."""
    from scipy.optimize import linprog
    n, scale = 2001, 1e6                                         # the error in units of 1e-6: the solver's tolerances are absolute
    f = 0.5 * np.cos(np.pi * (np.arange(n) + 0.5) / n)
    A, b, one = np.stack([f ** k * 2.0 ** -f for k in range(1, 6)], 1), 1 - 2.0 ** -f, np.ones((n, 1)) / scale
    fit = linprog([0] * 5 + [1], A_ub=np.block([[A, -one], [-A, -one]]), b_ub=np.concatenate([b, -b]), bounds=[(None, None)] * 6, method="highs",
                  options=dict(primal_feasibility_tolerance=1e-10, dual_feasibility_tolerance=1e-10))
    assert fit.status == 0
    ours = np.array(source[1][::-1])
    # coefficients in fp32, each moved by less than the fit's own error in its term
    assert np.abs((ours - fit.x[:5]) * 0.5 ** np.arange(1, 6)).max() < 2e-8
    assert np.abs(A @ fit.x[:5] - b).max() <= np.abs(A @ ours - b).max() < 1.2e-7


def _exp2_poly(x, coefficients):
    def fma(a, b, c):                                            # products of fp32 are exact in 64 bits
        return (a.astype(np.float64) * b.astype(np.float64) + np.float64(c)).astype(F)
    x = np.maximum(x, F(-127))
    t = x + F(12582912)
    f = (x.astype(np.float64) - (t - F(12582912))).astype(F)
    p = np.full_like(f, F(coefficients[0]))
    for c in coefficients[1:] + [1.0]:
        p = fma(p, f, F(c))
    return p * ((t.view(np.uint32) << np.uint32(23)) + np.uint32(0x3f800000)).view(F)


def test_error_is_the_stated_one(source):
    comment, coefficients = source
    assert re.search(r"at most 1\.8e-7", comment)
    top = np.arange(0x3e800000, 0x3f000001, dtype=np.uint32).view(F)           # every number of [1/4, 1/2], where the error is largest
    small = np.linspace(-0.25, 0.25, 4_000_001).astype(F)
    wide = np.linspace(-125.9, 8, 4_000_001).astype(F)
    for x in (top, -top, small, wide):
        e = _exp2_poly(x, coefficients).astype(np.float64) / np.exp2(x.astype(np.float64)) - 1
        assert np.abs(e).max() <= STATED
    below = np.array([-127, -128, -1e4, -3e38, -np.inf], F)
    assert (_exp2_poly(below, coefficients) == 0).all()
