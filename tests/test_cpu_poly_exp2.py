"""The polynomial exponential of the attention forward (`poly_exp2`), evaluated in float32 with the constants that stand in
its source: its error, and the exponents that have to become exactly 0."""
import os
import re

import numpy as np

import genesis_b200

SRC = os.path.join(os.path.dirname(genesis_b200.__file__), "csrc", "attention_common.cuh")
F = np.float32


def _constants():
    src = open(SRC).read()
    body = src[src.index("float2 poly_exp2(float2 x) {"):]
    body = body[:body.index("\n}")]
    num = r"(-?\d+\.\d*(?:e[+-]?\d+)?)f"
    clamp = {float(c) for c in re.findall(r'max\.NaN\.f32 [^;]*;" : "\+f"\(x\.[xy]\) : "f"\(' + num, body)}
    first = re.search(r"p = fma2\(f, make_float2\(" + num + r", [^)]*\), make_float2\(" + num, body)
    rest = re.findall(r"p = fma2\(p, f, make_float2\(" + num, body)
    magic = re.search(r"MAGIC = " + num + r" \+ " + num, body)
    assert len(clamp) == 1 and len(rest) == 4
    return clamp.pop(), [float(c) for c in (*first.groups(), *rest)], sum(float(c) for c in magic.groups())


def _fma(a, b, c):                          # (the product is exact in float64)
    return (a.astype(np.float64) * b.astype(np.float64) + np.asarray(c, np.float64)).astype(F)


def _poly_exp2(x):
    clamp, coef, magic = _constants()
    x = np.maximum(x.astype(F), F(clamp))
    u = x + F(magic)
    f = _fma(u - F(magic), np.full_like(x, -1), x)
    p = np.full_like(f, F(coef[0]))
    for c in coef[1:]:
        p = _fma(p, f, F(c))
    return p * (u.view(np.uint32) << np.uint32(23)).view(F)


def test_error_over_the_range_of_the_exponents():
    # differences of scores to a reference that may lie 8 below the maximum
    x = np.linspace(-126, 8, 2_000_001).astype(F)
    want = np.exp2(x.astype(np.float64))
    # 1.55e-7 of the polynomial and a rounding of 2^-24 each in the last fma and the product's input: below 2^-22
    assert float(np.abs(_poly_exp2(x) / want - 1).max()) <= 2.0 ** -22


def test_exponents_that_become_zero():
    assert not _poly_exp2(np.array([-np.inf, -3e38, -1e4, -128, -127, -126.5], F)).any()
    assert float(_poly_exp2(np.array([0.0], F))[0]) == 1.0 + 2.0 ** -23          # the constant term, 1.0000001192
