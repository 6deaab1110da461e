"""The polynomials of the flux sweep's erfc(x) and exp(-x^2) pair.

The coefficients are read from the device header and evaluated here in the
device's order of operations (fused steps emulated by extended precision),
against math.erfc and math.exp.  Bound: the argument reductions and the two
Horner schemes lose at most about 5 units of 2^-53 together, and math.erfc is
within 1; 6 and 4 units are allowed."""
import math
import os
import re

import numpy as np

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "gamera_cube_b200", "csrc", "gcs_physics.cuh")


def table(name):
    text = open(SOURCE).read()
    body = re.search(r"constexpr double %s\[\d+\] = \{(.*?)\};" % name, text, re.S).group(1)
    return [float(v) for v in body.replace("\n", " ").split(",")]


def fma(a, b, c):
    wide = np.longdouble
    return (wide(a) * wide(b) + wide(c)).astype(np.float64)


def erfc_exp(x):
    q, e = table("kQ"), table("kE")
    ax, y = np.abs(x), x * x
    low = fma(x, x, -y)
    shift = 6755399441055744.0
    fn = fma(-y, 1.4426950408889634, shift) - shift
    r = fma(-fn, 0.6931471805599453, -y)
    r = fma(-fn, 2.3190468138462996e-17, r) - low
    p = np.full_like(x, e[-1])
    for c in e[-2::-1]:
        p = fma(p, r, c)
    p = fma(p, r * r, r) + 1.0
    ex = np.where(y < 708.0, np.ldexp(p, fn.astype(int)), 0.0)
    s = ax + 4.0
    rs = 1.0 / s
    t = fma(-8.0, rs, 1.0)
    t = fma(fma(-t, s, ax - 4.0), rs, t)
    g = np.full_like(x, q[-1])
    for c in q[-2::-1]:
        g = fma(g, t, c)
    ec = ex * (g * rs)
    return np.where(x < 0.0, 2.0 - ec, ec), ex


def test_erfc_exp_pair():
    x = np.concatenate([np.linspace(-6.0, 6.0, 4001), np.linspace(6.0, 25.9, 1500),
                        [0.0, 1e-300, -1e-20, 1e-9]])
    ec, ex = erfc_exp(x)
    eps = 2.0 ** -53
    true_ec = np.array([math.erfc(v) for v in x])
    # exp(-x^2) with the rounding of x^2 taken into account
    y = x * x
    low = fma(x, x, -y)
    true_ex = np.array([math.exp(-a) * (1.0 - b) for a, b in zip(y, low)])
    assert np.max(np.abs(ec - true_ec) / true_ec) <= 6 * eps
    assert np.max(np.abs(ex - true_ex) / true_ex) <= 4 * eps


def test_beyond_the_range():
    ec, ex = erfc_exp(np.array([27.5, 40.0, -27.5, 300.0]))
    assert list(ex) == [0.0] * 4
    assert list(ec) == [0.0, 0.0, 2.0, 0.0]
