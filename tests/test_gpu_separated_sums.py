"""The separated pair sums (prefix moments over the smaller members) against the
oracle where they can go wrong: section counts around the tasks' 31 and 32 bins
and around the first separated lag, grids whose neighbour ratio leaves one or no
direct lag, populations that end or fall steeply within one section (those slots
keep the exact pair sum), single populated sections, signed vectors in the
Jacobian-vector product, and grids spanning hundreds of octaves.

Bound: |gpu - oracle| <= 1e-12 scale + 1e-280, the parity tests' bound. It covers
the rule's own allowance (a slot is separated where the left-out rounding of
x_j + x_k moves a bin by at most 2.5e-13 of its scale) and the sums' rounding
(some 30 roundings of 1.1e-16 a term)."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, agg_params, assert_close, gpu_agg, make_grid, oracle_agg, t

pytestmark = pytest.mark.gpu

SIZES = (2, 30, 31, 32, 33, 61, 62, 63, 64, 65, 93, 128, 129, 500)
GRIDS = {"q4": lambda n: pg.grids.geometric_pow2(n, 1e-21, 4.0),
         "q32": lambda n: pg.grids.geometric_pow2(n, 1e-21, 32.0),
         "q200": lambda n: pg.grids.geometric_pow2(n, 1e-21, 200.0),
         "ratio8": lambda n: 1e-100 * 8.0 ** np.arange(min(n, 200)),
         "irregular": lambda n: make_grid("generic", n, np.random.default_rng(n)),
         "irregular_wide": lambda n: 1e-20 * np.exp(np.cumsum(
             np.random.default_rng(n).uniform(0.05, 2.5, size=min(n, 130)))),
         "linear": lambda n: make_grid("linear", n, None)}


def populations(x, rng):
    n = len(x)
    z = np.log(x / x[n // 3])
    yield "smooth", np.exp(-0.5 * z * z) * 1e12
    N = np.exp(-0.5 * z * z) * 1e12
    N[n // 2:] = 0.0
    yield "cut", N
    yield "steep", 1e14 * np.exp(-3.0 * np.arange(n) * min(1.0, 150.0 / n))
    N = np.zeros(n)
    N[[0, n // 4, n // 2, (3 * n) // 4]] = (1e14, 1e10, 1e8, 1e3)
    yield "few", N


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_separated_sums_match_oracle(kernel, b0, bbr, bsh, grid):
    rng = np.random.default_rng(60 + kernel)
    cells = []
    for n in SIZES:
        x = GRIDS[grid](n)
        for what, N in populations(x, rng):
            ref, scale, _ = oracle_agg(N, x, agg_params(len(x), kernel, b0, bbr, bsh))
            cells.append((x, N, ref, scale, "k=%d %s n=%d %s" % (kernel, grid, len(x), what)))
            for mode in (pg.MODE_GATHER, pg.MODE_SCATTER):
                p = agg_params(len(x), kernel, b0, bbr, bsh, x, geometric=not grid.startswith(("irr", "lin")))
                code, got = gpu_agg(N, x, p, mode)
                assert code == 0
                assert_close(got, ref, scale, "single mode %d " % mode + cells[-1][4])
    # the same as cells of one plan, each on its own grid
    with pg.BatchPlan([c[0] for c in cells], [len(c[0]) for c in cells], range(len(cells)), kernel) as plan:
        rhs = t(np.zeros(plan.total))
        prm = t(pg.batch.cell_params(len(cells), beta0=b0, beta_br=bbr, beta_sh=bsh))
        assert plan.rhs(t(np.concatenate([c[1] for c in cells])), rhs, prm) == 0
        for got, (x, N, ref, scale, what) in zip(plan.split(rhs.cpu().numpy()), cells):
            assert_close(got, ref, scale, "batched " + what)


@pytest.mark.parametrize("grid", ["q4", "q32", "irregular", "linear"])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_separated_jvp_matches_oracle(kernel, b0, bbr, bsh, grid):
    rng = np.random.default_rng(80 + kernel)
    cells = []
    for n in SIZES:
        x = GRIDS[grid](n)
        for what, N in populations(x, rng):
            v = rng.standard_normal(len(x)) * np.maximum(N, 1e-3 * N.max())
            ref, scale, _ = pyoracle.aggregation_rhs_jvp(N, v, x, kernel, b0, bbr, bsh)
            cells.append((x, N, v, ref, scale, "k=%d %s n=%d %s" % (kernel, grid, len(x), what)))
    # one cell alone (a cluster per cell and several warps per task), then all
    for group in ([cells[-1]], cells):
        with pg.BatchPlan([c[0] for c in group], [len(c[0]) for c in group], range(len(group)), kernel) as plan:
            out = t(np.zeros(plan.total))
            prm = t(pg.batch.cell_params(len(group), beta0=b0, beta_br=bbr, beta_sh=bsh))
            assert plan.jvp(t(np.concatenate([c[1] for c in group])), t(np.concatenate([c[2] for c in group])),
                            out, prm) == 0
            for got, (x, N, v, ref, scale, what) in zip(plan.split(out.cpu().numpy()), group):
                assert_close(got, ref, scale, "jvp " + what)


@pytest.mark.parametrize("n,q", [(497, 64.0), (641, 64.0), (700, 512.0), (1500, 128.0), (3000, 256.0)])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_window_sums_match_oracle(kernel, b0, bbr, bsh, n, q):
    """Fine grids, where runs of lags with one bracket offset are summed by window
    tables: windows within a block of 64 bins, across one edge and across whole
    blocks, cut at bin 0; a grid that ends before the lags that land on their larger
    member (n = 700, q = 512); populations the windows' rounding rule rejects, and
    one with a negative entry (no windows at all)."""
    rng = np.random.default_rng(90 + kernel)
    x = pg.grids.geometric_pow2(n, 1e-21, q)
    p = agg_params(n, kernel, b0, bbr, bsh, x)
    for what, N in [*populations(x, rng), ("sparse", np.where(np.arange(n) % 97 == 5, 1e9, 0.0)),
                    ("negative", -np.abs(rng.standard_normal(n)) + 0.5)]:
        ref, scale, _ = oracle_agg(N, x, p)
        for mode in (pg.MODE_GATHER, pg.MODE_SCATTER):
            code, got = gpu_agg(N, x, p, mode)
            assert code == 0
            assert_close(got, ref, scale, "k=%d n=%d q=%g %s mode %d" % (kernel, n, q, what, mode))


@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_window_sums_keep_a_populations_foot(kernel, b0, bbr, bsh):
    """A population that falls to 1e-305 on a fine grid: bins that receive down to 1e-303
    keep the relative bound of the others (1e-12 of their sum of |terms|, no floor): the
    breakage guard N > 2.2e-308 and its adjoint see such values grow from nothing."""
    n = 1500
    x = pg.grids.geometric_pow2(n, 1e-21, 128.0)
    p = agg_params(n, kernel, b0, bbr, bsh, x)
    for c, width in ((300, 24.0), (500, 16.0)):
        N = 1e12 * np.exp(-0.5 * ((np.arange(n) - c) / width) ** 2)
        N[N < 1e-305] = 0.0
        ref, scale, _ = oracle_agg(N, x, p)
        code, got = gpu_agg(N, x, p, pg.MODE_GATHER)
        assert code == 0
        foot = (scale > 1e-303) & (scale < 1e-200)
        assert foot.sum() > 10
        err = np.abs(got - ref)[foot] / scale[foot]
        assert err.max() <= 1e-12, (kernel, c, err.max())
