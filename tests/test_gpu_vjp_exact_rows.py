"""VJP rows that keep their exact pair sums: a lambda that is nonzero only where a
population has ended makes nearly every row one of them, and then all lags are summed
pair by pair. Against the oracle (the VJP tests' bound, 1e-12 of an entry's sum of
|terms|), and their time against an ordinary lambda's."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, agg_params, assert_close, dev, t

pytestmark = pytest.mark.gpu


def cases(n):
    i = np.arange(n)
    N = 1e12 * np.exp(-0.5 * ((i - n / 3.0) / (n / 12.0 + 1.0)) ** 2)
    N[n // 2:] = 0.0
    yield "above the population", N, (i >= n // 2) * 1.0
    yield "one section above", N, (i == n // 2) * 1.0
    M = np.where(i % 2 == 0, N, 0.0)
    yield "an empty section", M, (i == 2 * (n // 6) + 1) * 1.0
    yield "empty sections", M, (i % 2 == 1) * np.cos(i)
    yield "top section", N, (i == n - 1) * 1.0
    yield "ordinary", N, np.cos(0.7 * i)


@pytest.mark.parametrize("n,q", [(33, 4.0), (64, 4.0), (129, 8.0), (300, 4.0), (300, 32.0), (520, 128.0), (960, 32.0)])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_exact_rows_match_oracle(kernel, b0, bbr, bsh, n, q):
    import torch

    x = pg.grids.geometric_pow2(n, 1e-21, q)
    p = agg_params(n, kernel, b0, bbr, bsh, x)
    prm = pg.batch.cell_params(1, beta0=b0, beta_br=bbr, beta_sh=bsh)
    for what, N, lam in cases(n):
        gN, gp, sN, sp, _ = pyoracle.aggregation_rhs_vjp(N, x, lam, kernel, b0, bbr, bsh, with_scale=True)
        g, h = torch.zeros(n, dtype=torch.float64, device=dev()), torch.zeros(3, dtype=torch.float64, device=dev())
        pg.check(pg.aggregation_rhs_vjp(t(N), t(x), t(lam), g, h, p))
        name = "k=%d n=%d q=%g %s" % (kernel, n, q, what)
        assert_close(g.cpu().numpy(), gN, sN, name)
        assert_close(h.cpu().numpy(), gp, sp, name + " parameters")
        # as a plan of one cell (row tiles) and of many (blocks of rows)
        for cells in (1, 96):
            if cells > 1 and what not in ("above the population", "an empty section"):
                continue
            with pg.BatchPlan([x], [n] * cells, [0] * cells, kernel) as plan:
                G = torch.zeros(plan.total, dtype=torch.float64, device=dev())
                H = torch.zeros(cells, 8, dtype=torch.float64, device=dev())
                pg.check(plan.rhs_vjp(t(np.tile(N, cells)), t(np.tile(lam, cells)), G, H, t(np.tile(prm, (cells, 1)))))
                G, H = G.cpu().numpy().reshape(cells, n), H.cpu().numpy()
            assert (G == G[0]).all() and (H == H[0]).all(), name
            assert_close(G[0], gN, sN, name + " cells %d" % cells)
            assert_close(H[0, :3], gp, sp, name + " cells %d parameters" % cells)


@pytest.mark.parametrize("n,q", [(64, 4.0), (300, 4.0), (960, 32.0)])
def test_exact_rows_take_no_multiple_of_an_ordinary_call(n, q):
    """One exact row after the other took 8 times an ordinary lambda's time; all lags
    pair by pair 1.3 times."""
    import torch

    x = pg.grids.geometric_pow2(n, 1e-21, q)
    p = agg_params(n, 5, 0.0, 6.73e-18, 66.67, x)
    us = {}
    for what, N, lam in cases(n):
        if what not in ("above the population", "ordinary"):
            continue
        a = [t(N), t(x), t(lam)]
        g, h = torch.zeros(n, dtype=torch.float64, device=dev()), torch.zeros(3, dtype=torch.float64, device=dev())
        ts = []
        for r in range(26):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            pg.check(pg.aggregation_rhs_vjp(*a, g, h, p))
            e1.record()
            e1.synchronize()
            ts.append(e0.elapsed_time(e1))
        us[what] = float(np.median(ts[5:]))
    assert us["above the population"] <= 3.0 * us["ordinary"], us
