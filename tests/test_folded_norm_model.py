"""The error model of folded norms, on the CPU: the tensor core sums the products and the
three pieces of -|b|^2 / 2 (columns d .. d + 2) with the truncating accumulation of
tests/test_tc_error_model.py, and the estimate |a|^2 - 2 w stays within the bound that
the engine takes for it, c_rel (|a|^2 + |b|^2) + c_abs, on random, cancelling and
unevenly scaled points."""
import math

import numpy as np
import pytest

from test_tc_error_model import tc_dot, tf32_rn


def round_op(form, v):
    return v.astype(np.float16).astype(np.float64) if form == "fp16" else tf32_rn(v.astype(np.float32)).astype(
        np.float64)


def pieces(form, v):
    """v in three operand elements and the scales that the A side holds for them."""
    scales = (2.0 ** 15, 2.0 ** 4, 2.0 ** -7) if form == "fp16" else (1.0, 1.0, 1.0)
    out, rest = [], v
    for s in scales:
        m = round_op(form, rest / s)
        out.append(m)
        rest = rest - m * s
    return np.stack(out, 1), np.array(scales), rest


def bound(form, d):
    kstep = 16 if form == "fp16" else 8
    terms = 2 * (-(-(d + 3) // kstep) * kstep)  # the pieces double the sum of magnitudes
    u = 2.0 ** -11
    c_rel = 1.25 * (2 * u + u * u + 2 * 2.0 ** -24 + terms * 2.0 ** -22 + 12 * 2.0 ** -24 + d * 2.0 ** -50)
    c_abs = 1.25 * (d * 2.0 ** -13 + 2.0 ** -31) if form == "fp16" else 1e-30
    return c_rel, c_abs


@pytest.mark.parametrize("form", ["fp16", "tf32"])
@pytest.mark.parametrize("d", [1, 4, 13, 29, 61, 125, 253])
@pytest.mark.parametrize("k", [2, 4, 8, 16])
def test_estimate_within_the_bound(form, d, k):
    rng = np.random.default_rng(31 * d + k)
    n = 300
    a = rng.uniform(-1, 1, (n, d))
    b = np.concatenate([a[:100] * (1 + 2.0 ** -9 * rng.standard_normal((100, d))),  # near pairs: s cancels
                        -a[100:200],                                                 # the far end of the range
                        rng.uniform(-1, 1, (100, d)) * np.exp(rng.uniform(-8, 0, (100, d)))])
    scale = 2.0 ** 9 / max(np.abs(a).max(), np.abs(b).max()) if form == "fp16" else 1.0
    scale = 2.0 ** math.floor(math.log2(scale))
    if form == "tf32":  # TF32 operands come from the FP32 value
        a, b = (v.astype(np.float32).astype(np.float64) for v in (a, b))
    A, B = a * scale, b * scale
    nb = (B * B).sum(1)
    m, s, rest = pieces(form, 0.5 * nb)
    assert (np.abs(rest) <= 2.0 ** -33 * 0.5 * nb + 2.0 ** -32).all()
    prods = np.concatenate([round_op(form, A) * round_op(form, B), -m * s], axis=1)
    kstep = 16 if form == "fp16" else 8
    prods = np.pad(prods, ((0, 0), (0, -prods.shape[1] % kstep)))
    w = tc_dot(prods, k).astype(np.float32)
    na = (A * A).sum(1)
    est = (na.astype(np.float32) + np.float32(-2) * w).astype(np.float64)
    exact = ((A - B) ** 2).sum(1)
    c_rel, c_abs = bound(form, d)
    err = np.abs(est - exact)
    ratio = (err / (c_rel * (na + nb) + c_abs)).max()
    print(f"{form} d={d} k={k}: max |est - dist2| / bound = {ratio:.3f}")
    assert ratio <= 1.0 and err.max() > 0
