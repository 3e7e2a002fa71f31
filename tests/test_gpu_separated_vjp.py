"""The VJP's separated sums (lags whose pairs land on their larger member) against
the oracle's adjoint: section counts around the row blocks of 32 and the scan
blocks of 64, grids with one or no direct lag, populations that end or fall
steeply, and smooth, random, one-hot and step-shaped lambda (where a row's whole
sum can be a few tiny weights, whose rounding then counts).

Bound: |gpu - oracle| <= 1e-12 scale + 1e-280 (the VJP tests' bound); the rule's
own allowance is 5e-13 of a row's scale."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, agg_params, assert_close, t
from test_gpu_separated_sums import GRIDS, populations
from test_gpu_vjp import gpu_agg_vjp

pytestmark = pytest.mark.gpu

SIZES = (2, 31, 32, 33, 64, 65, 129, 400)


def lambdas(x, rng):
    n = len(x)
    yield "power", (x / x[n // 2]) ** (2.0 / 3.0)
    yield "random", rng.standard_normal(n)
    one = np.zeros(n)
    one[n // 2] = 1.0
    yield "one", one
    yield "step", (np.arange(n) >= (2 * n) // 3).astype(float)


@pytest.mark.parametrize("grid", ["q4", "q32", "q200", "ratio8"])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_separated_vjp_matches_oracle(kernel, b0, bbr, bsh, grid):
    rng = np.random.default_rng(40 + kernel)
    for n in SIZES:
        x = GRIDS[grid](n)
        for what, N in populations(x, rng):
            for lwhat, lam in lambdas(x, rng):
                p = agg_params(len(x), kernel, b0, bbr, bsh, x)
                code, gN, gp = gpu_agg_vjp(N, x, lam, p)
                assert code == 0
                rN, rp, sN, sp, _ = pyoracle.aggregation_rhs_vjp(N, x, lam, kernel, b0, bbr, bsh, p.log_x0,
                                                                 p.inv_log_r, exact_bracket=True, with_scale=True)
                tag = "k=%d %s n=%d %s lambda %s" % (kernel, grid, len(x), what, lwhat)
                assert_close(gN, rN, sN, "dL/dN " + tag)
                assert_close(gp, rp, sp, "dL/dbeta " + tag)


@pytest.mark.parametrize("grid", ["q4", "q32", "q200", "ratio8", "irregular"])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_batched_separated_vjp_matches_oracle(kernel, b0, bbr, bsh, grid):
    """The batched row blocks: the same populations and lambdas as cells of one plan,
    and one cell alone (a cluster of prep CTAs and several warps per block)."""
    rng = np.random.default_rng(140 + kernel)
    cells = []
    for n in SIZES:
        x = GRIDS[grid](n)
        for what, N in populations(x, rng):
            for lwhat, lam in lambdas(x, rng):
                ref = pyoracle.aggregation_rhs_vjp(N, x, lam, kernel, b0, bbr, bsh, exact_bracket=True,
                                                   with_scale=True)
                cells.append((x, N, lam, ref, "k=%d %s n=%d %s lambda %s" % (kernel, grid, len(x), what, lwhat)))
    for group in ([cells[-4]], cells):
        with pg.BatchPlan([c[0] for c in group], [len(c[0]) for c in group], range(len(group)), kernel) as plan:
            prm = t(pg.batch.cell_params(len(group), beta0=b0, beta_br=bbr, beta_sh=bsh))
            gN, gp = t(np.zeros(plan.total)), t(np.zeros((len(group), 8)))
            assert plan.rhs_vjp(t(np.concatenate([c[1] for c in group])), t(np.concatenate([c[2] for c in group])),
                                gN, gp, prm) == 0
            gp = gp.cpu().numpy()
            for c, (got, (x, N, lam, ref, what)) in enumerate(zip(plan.split(gN.cpu().numpy()), group)):
                rN, rp, sN, sp, _ = ref
                assert_close(got, rN, sN, "batched dL/dN " + what)
                assert_close(gp[c, :3], rp, sp, "batched dL/dbeta " + what)
