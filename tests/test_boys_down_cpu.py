"""The evaluation of the quartet kernels' Boys values (boys_down, csrc/pfe_common.cuh):
the top order from the tabulated point nearest T, e^-T from its tabulated value and a
short series, the lower orders by downward recursion -- restated here in FP64 on the
host's IGAMMA table and checked against the incomplete gamma function over each top
order's range.

Tolerance: the series leave 0.025^7/7! F_{m+7} < 2e-15 F_m and 4e-18, and every step of
the stable downward recursion rounds twice: 1e-14 relative covers orders up to 8.
"""
import math

import numpy as np
import pytest
from scipy import special

from polymer_b200 import system

TF = [33, 37, 41, 43, 46, 49, 51, 54, 56]


def _exact(m, t):
    # F_m(T) = Gamma(m + 1/2) P(m + 1/2, T) / (2 T^(m + 1/2)), the series near T = 0
    if t < 1e-3:
        return sum((-t) ** k / (math.factorial(k) * (2 * m + 2 * k + 1)) for k in range(6))
    return special.gamma(m + 0.5) * special.gammainc(m + 0.5, t) / (2.0 * t ** (m + 0.5))


def _boys_down(L, t, tab):
    ts = int(math.floor(t * 20.0 + 0.5))
    h = 0.05 * ts - t
    f = 0.0
    for k in range(6, -1, -1):
        f = f * h + tab[ts, L + k] / math.factorial(k)
    x = 0.0
    for k in range(7, -1, -1):
        x = x * h + 1.0 / math.factorial(k)
    e = math.exp(-0.05 * ts) * x
    out = [0.0] * (L + 1)
    out[L] = f
    for m in range(L - 1, -1, -1):
        out[m] = (2.0 * t * out[m + 1] + e) / (2 * m + 1)
    return out


@pytest.mark.parametrize('L', range(9))
def test_top_order_and_downward_recursion_match_the_incomplete_gamma_function(L):
    tab = system.fmt_table()
    rng = np.random.default_rng(L)
    edges = [0.0, 1e-9, 0.0249999, 0.025, 0.0250001, TF[L] - 0.0250001, TF[L] - 1e-12]
    for t in edges + list(rng.uniform(0.0, TF[L], 400)):
        got = _boys_down(L, t, tab)
        for m in range(L + 1):
            ref = _exact(m, t)
            assert abs(got[m] - ref) <= 1e-14 * ref, (L, m, t)
