"""Aggregation coefficients of either sign (a user's kernel fit may pass through one): the
rules that decide which pairs are summed exactly compare sums of rates, so they must not
turn round with the sign.

All coefficients negated: every sum changes its sign and nothing else, so the result is
the negative bit for bit. Coefficients of opposite signs: the parity bound, 1e-12 of a
bin's sum of |terms|, with the terms of the two parts counted apart (their sums are
formed apart)."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, agg_params, assert_close, gpu_agg, t

pytestmark = pytest.mark.gpu


def populations(x):
    n = len(x)
    z = np.arange(n) - n // 3
    yield "smooth", 1e12 * np.exp(-0.5 * (z / (n / 20.0)) ** 2)
    yield "narrow", np.where(np.abs(z) < n // 12, 1e12 * np.exp(-0.5 * (z / 3.0) ** 2), 0.0)
    yield "sparse", np.where(np.arange(n) % 97 == 5, 1e9, 0.0)
    yield "steep", 1e14 * np.exp(-3.0 * np.arange(n) * min(1.0, 150.0 / n))
    N = np.zeros(n)
    N[[0, n // 4, n // 2, (3 * n) // 4]] = (1e14, 1e10, 1e8, 1e3)
    yield "few", N


@pytest.mark.parametrize("n,q", [(64, 4.0), (400, 64.0), (1500, 128.0), (3000, 256.0)])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_negated_coefficients_negate_the_result(kernel, b0, bbr, bsh, n, q):
    x = pg.grids.geometric_pow2(n, 1e-21, q)
    for what, N in populations(x):
        out = []
        for s in (1.0, -1.0):
            code, got = gpu_agg(N, x, agg_params(n, kernel, s * b0, s * bbr, s * bsh, x), pg.MODE_GATHER)
            assert code == 0
            out.append(got)
        assert np.array_equal(out[0], -out[1]), (what, int((out[0] != -out[1]).sum()))


@pytest.mark.parametrize("n,q", [(400, 64.0), (1500, 128.0)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_opposite_signs_match_oracle(sign, n, q):
    x = pg.grids.geometric_pow2(n, 1e-21, q)
    bbr, bsh = sign * 6.73e-18, -sign * 66.67
    for what, N in populations(x):
        a, sa, _ = pyoracle.aggregation_rhs(N, x, 3, 0.0, bbr, 0.0, 0.0, 0.0, exact_bracket=True)
        b, sb, _ = pyoracle.aggregation_rhs(N, x, 4, 0.0, 0.0, bsh, 0.0, 0.0, exact_bracket=True)
        code, got = gpu_agg(N, x, agg_params(n, 5, 0.0, bbr, bsh, x), pg.MODE_GATHER)
        assert code == 0
        assert_close(got, a + b, np.abs(sa) + np.abs(sb), "%s n=%d" % (what, n))
