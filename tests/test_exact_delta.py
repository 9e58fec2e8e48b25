"""The difference n x - sum(v) of floats that the outer operator forms on the
FP32 pipe (dfl::exact_delta), restated with numpy's IEEE floats, against exact
rationals: its error stays at one FP64 rounding of the result and, scaled by
T S as the operator scales it, below that of the FP64 sum of products it
stands for, on smooth, rough and widely spread values."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def two_sum(a, b):
    s = f32(a + b)
    ap = f32(s - b)
    bp = f32(s - ap)
    return s, f32(f32(a - ap) + f32(b - bp))


def exact_delta(n, x, v):
    p = f32(f32(n) * x)
    pe = f32(float(n) * float(x) - float(p))  # the fused multiply-add's exact error
    s, e = two_sum(v[0], v[1])
    err, rest = e, f32(0)

    def more(e):
        nonlocal err, rest
        err, lo = two_sum(err, e)
        rest = f32(rest + lo)
    for d in range(1, len(v) // 2):
        a, al = two_sum(v[2 * d], v[2 * d + 1])
        s, ql = two_sum(s, a)
        more(al)
        more(ql)
    h, hl = two_sum(p, f32(-s))
    more(f32(-pe))
    lo, ll = two_sum(hl, f32(-err))
    return float(h) + float(lo) + float(f32(ll - rest))


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


VALUES = {
    "smooth": lambda g, k: (1 + 1e-3 * g.standard_normal(k)) * g.standard_normal(),
    "rough": lambda g, k: g.standard_normal(k),
    "spread": lambda g, k: g.standard_normal(k) * 10.0 ** g.uniform(-12, 2, k),
    "zeros": lambda g, k: g.standard_normal(k) * g.integers(0, 2, k),
}


@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("kind", VALUES)
def test_error_of_the_exact_difference(kind, nd):
    g = np.random.default_rng(7)
    new, old = [], []
    for _ in range(150):
        w = VALUES[kind](g, 2 * nd + 1).astype(f32)
        x, v = w[0], w[1:]
        n = 2 * nd + int(g.integers(-1, 2))  # a Neumann or Dirichlet face among them
        if n != 2 * nd:
            v[0] = 0
        T, S = float(g.uniform(1e-3, 1)), 1 / float(g.uniform(1e-6, 1e-2))
        exact = n * Fraction(float(x)) - sum(Fraction(float(q)) for q in v)
        d = exact_delta(n, x, v)
        # one rounding of the result and what the dropped bits below 2^-70 give
        assert abs(Fraction(d) - exact) <= abs(exact) * Fraction(2) ** -53 + Fraction(float(abs(w).max())) * Fraction(2) ** -69
        exact = exact * Fraction(T) * Fraction(S)
        P, off = 0.0, 0.0
        for _q in range(n):
            P += T
        for q in v:
            off = fma(T, float(q), off)
        scale = float(Fraction(T) * Fraction(S)) * n * max(float(abs(w).max()), 1e-300)
        new.append(float(Fraction((T * S) * d) - exact) / scale)
        old.append(float(Fraction(fma(float(x), P * S, -(off * S))) - exact) / scale)
    rms = lambda a: float(np.sqrt(np.mean(np.square(a))))  # noqa: E731
    # two roundings of T S d against at least as many of larger terms; equal
    # where a single term dominates (spread), hence the sampling margin
    assert rms(new) <= 1.25 * rms(old)
