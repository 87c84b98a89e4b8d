"""The sine of the insertions' window (noa_b200/csrc/fp_common.cuh, sinpi_reduced and, on pairs, WindowPair): its
steps in single precision, with the coefficients the kernels compile, against the sine in double precision."""

import pathlib
import re

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "noa_b200" / "csrc"
F = np.float32


def coefficients():
    text = (CSRC / "fp_common.cuh").read_text()
    terms = re.search(r"#define NB_SINPI \{([^}]*)\}", text).group(1)
    rounding = re.search(r"SINPI_ROUND = ([0-9.]+)f;", text).group(1)
    return [F(c.strip().rstrip("f")) for c in terms.split(",")], F(rounding)


def fma(a, b, c):  # the product of two floats is exact in a double, whose sum is then rounded to a float
    return (a.astype(np.float64) * b + c).astype(F)


def sinpi(s):
    c, rounding = coefficients()
    t = s + rounding
    r = s - (t - rounding)
    u = r * r
    p = fma(u, c[0], c[1])
    for k in range(2, 5):
        p = fma(u, p, c[k])
    odd = (t.view(np.int32) & 1).astype(bool)
    return np.where(odd, -(r * p), r * p)


@pytest.mark.parametrize("lowest, highest", [(0., 0.5), (0.5, 8.), (8., 4096.), (4096., 2.0 ** 21)])
def test_sine_of_the_window(lowest, highest):
    """The phase is reduced exactly; the rounded coefficients give 2.4e-8, the product 2^-24, u's rounding and the
    last two steps of the polynomial at most 2^-24 each: 2.4e-8 + 3 * 6e-8 = 2.1e-7 of the sine."""
    s = np.random.default_rng(7).uniform(lowest, highest, 200_000).astype(F)
    s = np.concatenate([s, np.round(s), np.round(s) + F(0.5), F([lowest, highest])])
    got, k = sinpi(s).astype(np.float64), np.round(s.astype(np.float64))
    want = np.sin(np.pi * (s - k)) * np.where(k % 2, -1., 1.)
    assert np.all(got[want == 0] == 0)
    error = np.abs(got - want)[want != 0] / np.abs(want[want != 0])
    assert error.max() <= 2.1e-7
    assert np.sqrt(np.mean(error ** 2)) <= 6e-8
