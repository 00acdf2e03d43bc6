"""The FP64 sweep's table-driven exponential: its coefficients and table on the
CPU, and its values on the GPU through the self-excitation probabilities."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "hawkes_b200", "csrc", "hphc_sweep.cuh")


def _constants():
    text = open(SRC).read()
    c = [float.fromhex(re.search(rf"kE{k} = (0x[0-9a-fp.+-]+);", text).group(1))
         for k in range(1, 6)]
    table = re.search(r"kExpTable\[32\] = \{(.*?)\};", text, re.S).group(1)
    return c, [float.fromhex(v) for v in table.replace("\n", " ").split(",") if v.strip()]


def test_polynomial_and_table():
    c, table = _constants()
    ld = np.longdouble
    f = np.linspace(-0.5, 0.5, 200001).astype(ld)
    q = np.zeros_like(f)
    for v in reversed(c):
        q = q * f + ld(v)
    exact = np.exp2(f / 32)
    rel = (1 + f * q - exact) / exact
    assert np.max(np.abs(rel)) <= 2.0 ** -53  # half a unit in the last place
    assert abs(np.mean(rel)) <= 5e-18
    want = np.exp2(np.arange(32, dtype=ld) / 32)
    assert np.array_equal(np.array(table), want.astype(np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 127, 129, 400])
def test_values_through_the_probabilities(n):
    # One dimension, equal locations: event i's self-excitation terms are
    # exp(-omega (t_i - t_j)), its background terms exp(-b^2 dt^2 / 2) with b
    # so large that only B_ii is left, so P_i shows the exponentials over the
    # whole range.  A sum of positive terms, each within 1.5 units in the last
    # place (table 1/2, product 1/2, polynomial and exponent under 1/2) plus
    # the exponent's own rounding, 2 units of |x| relative: 2e-16 (2 + 2 * 710)
    # at the far end, and about 1e-15 for the P_i formed from it.
    import hawkes_b200 as hb
    rng = np.random.default_rng(n)
    t = np.sort(rng.uniform(0.0, 720.0, size=n))
    t[0], t[-1] = 0.0, 720.0
    loc = np.zeros((n, 1))
    p = np.array([1.0, 1.0, 1e6, 1.0, 1.0, 1.0])
    with hb.CudaHawkes(1, n, hb.CUDA, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        got = e.getProbsSelfExcite()
    dt = (t[:, None] - t[None, :]).astype(np.longdouble)
    S = np.where(dt > 0, np.exp(-np.abs(dt)), 0).sum(1) / np.sqrt(2 * np.longdouble(np.pi))
    B = np.longdouble(1e6) / (2 * np.longdouble(np.pi))
    want = S / (B + S)
    big = want > 1e-290
    assert np.all(np.abs(got[big] - want[big]) <= 3.2e-13 * want[big])
    near = want > 1e-20
    assert np.all(np.abs(got[near] - want[near]) <= 3e-14 * want[near])
    assert np.all((got[~big] >= 0) & (got[~big] <= 1e-289))
