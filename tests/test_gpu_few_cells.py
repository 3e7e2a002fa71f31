"""Plans of few cells: tasks spread over the SMs, blocks of rows or row tiles in the VJP,
and the foot of a population in the batched prefix sums."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, assert_close, dev, make_grid, oracle_agg, agg_params, t

pytestmark = pytest.mark.gpu


def _plan(n, q, cells, kernel=5):
    x = pg.grids.geometric_pow2(n, 1e-21, q) if q else make_grid("linear", n, None)
    return pg.BatchPlan([x], [n] * cells, [0] * cells, kernel)


def test_few_tasks_get_an_sm_each():
    """Tasks that share a CTA share its SM's FP64 pipe: no two do while SMs are idle."""
    for n, q, cells in ((31, 0.0, 16), (31, 4.0, 16), (100, 4.0, 8), (200, 32.0, 1), (960, 4.0, 1)):
        with _plan(n, q, cells) as plan:
            _, bundles = plan.schedule()
            assert bundles == cells * ((n + 30) // 31), (n, q, cells, bundles)


def test_few_tasks_get_more_warps():
    """A task's chain of latencies is shorter with more warps, whatever its direct lags."""
    for n, q, cells, least in ((31, 4.0, 1, 256), (200, 4.0, 1, 256), (31, 0.0, 16, 256), (100, 4.0, 128, 128)):
        with _plan(n, q, cells) as plan:
            sizes, _ = plan.schedule()
            assert min(sizes.values()) >= least, (n, q, cells, sizes)
    with _plan(100, 4.0, 4096) as plan:               # and a warp each where the SMs are full
        sizes, _ = plan.schedule()
        assert set(sizes.values()) == {32}, sizes


@pytest.mark.parametrize("cells", [1, 3, 40, 200])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_rhs_and_vjp_match_oracle(kernel, b0, bbr, bsh, cells):
    """Counts of cells on either side of the rules, cells of uneven lengths on one grid
    each of four kinds."""
    import torch

    rng = np.random.default_rng(cells + 10 * kernel)
    kinds = [pg.grids.geometric_pow2(130, 1e-21, 4.0), pg.grids.geometric_pow2(200, 1e-21, 32.0),
             make_grid("linear", 90, None), make_grid("generic", 140, rng)]
    which = [c % 4 for c in range(cells)]
    cell_n = [int(len(kinds[w]) - (c * 7) % 60) for c, w in enumerate(which)]
    Ns = [1e12 * np.exp(-0.5 * ((np.arange(n) - n / 3.0) / (n / 9.0)) ** 2) for n in cell_n]
    ls = [rng.standard_normal(n) for n in cell_n]
    with pg.BatchPlan(kinds, cell_n, which, kernel) as plan:
        prm = t(pg.batch.cell_params(cells, beta0=b0, beta_br=bbr, beta_sh=bsh))
        N, lam = t(np.concatenate(Ns)), t(np.concatenate(ls))
        out, gN = torch.zeros_like(N), torch.zeros_like(N)
        gp = torch.zeros(cells, 8, dtype=torch.float64, device=dev())
        pg.check(plan.rhs(N, out, prm))
        pg.check(plan.rhs_vjp(N, lam, gN, gp, prm))
        outs, gNs, gp = plan.split(out.cpu().numpy()), plan.split(gN.cpu().numpy()), gp.cpu().numpy()
    for c in range(min(cells, 12)):
        x = kinds[which[c]][:cell_n[c]]
        ref, scale, _ = oracle_agg(Ns[c], x, agg_params(cell_n[c], kernel, b0, bbr, bsh))
        assert_close(outs[c], ref, scale, "rhs cell %d of %d" % (c, cells))
        g, p, sg, sp, _ = pyoracle.aggregation_rhs_vjp(Ns[c], x, ls[c], kernel, b0, bbr, bsh, with_scale=True)
        assert_close(gNs[c], g, sg, "vjp cell %d of %d" % (c, cells))
        assert_close(gp[c, :3], p, sp, "vjp parameters cell %d of %d" % (c, cells))


@pytest.mark.parametrize("cells", [1, 64])
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_cells_keep_a_populations_foot(kernel, b0, bbr, bsh, cells):
    """As the single instances' tests: bins that receive down to 1e-290 keep 1e-12 of
    their sum of |terms|, no floor."""
    import torch

    for n, q in ((60, 4.0), (300, 32.0), (700, 128.0)):
        x = pg.grids.geometric_pow2(n, 1e-21, q)
        p = agg_params(n, kernel, b0, bbr, bsh, x)
        N = 1e12 * np.exp(-0.5 * ((np.arange(n) - n // 4) / max(0.7, n / 100.0)) ** 2)
        N[N < 1e-305] = 0.0
        ref, scale, _ = oracle_agg(N, x, p)
        with pg.BatchPlan([x], [n] * cells, [0] * cells, kernel) as plan:
            prm = t(pg.batch.cell_params(cells, beta0=b0, beta_br=bbr, beta_sh=bsh))
            y = t(np.tile(N, cells))
            out = torch.zeros_like(y)
            pg.check(plan.rhs(y, out, prm))
            got = out.cpu().numpy().reshape(cells, n)
        foot = (scale > 1e-290) & (scale < 1e-200)
        assert foot.sum() >= 3
        err = np.abs(got - ref)[:, foot] / scale[foot]
        assert err.max() <= 1e-12, (kernel, n, err.max())


def test_one_cells_vjp_keeps_up_with_an_irregular_one():
    """One cell of 960 sections at 128 an octave: by blocks of rows 1.6 times a cell on an
    irregular grid (row tiles), 0.8 by tiles."""
    import torch

    us = []
    for x in (pg.grids.geometric_pow2(960, 1e-21, 128.0), make_grid("generic", 960, np.random.default_rng(960))):
        N = t(1e12 * np.exp(-0.5 * ((np.arange(960) - 320) / 80.0) ** 2))
        lam = t(np.random.default_rng(3).standard_normal(960))
        with pg.BatchPlan([x], [960], [0], 5) as plan:
            prm = t(pg.batch.cell_params(1, beta_br=6.73e-18, beta_sh=66.67))
            gN, gp = torch.zeros_like(N), torch.zeros(1, 8, dtype=torch.float64, device=dev())
            ts = []
            for r in range(30):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                pg.check(plan.rhs_vjp(N, lam, gN, gp, prm))
                e1.record()
                e1.synchronize()
                ts.append(e0.elapsed_time(e1))
        us.append(float(np.median(ts[5:])))
    assert us[0] <= 1.2 * us[1], us
