"""RK4 of plans whose cells are all small: every step of a call in one launch, a CTA
per cell (batch_cells_rk4). Against the oracle's rk4_step cell by cell, with the bound of
the other batched RK4 tests (1e-11 of the state, rounding of 4 stages a step)."""
import numpy as np
import pytest

import pbe_gb300 as pg
import pyoracle
from gpu_util import AGG_KERNELS, make_grid, t

pytestmark = pytest.mark.gpu

# edges of the 31-bin slot blocks, the smallest cells and the largest plan (4 blocks)
SIZES = [1, 2, 3, 30, 31, 32, 33, 61, 62, 63, 93, 94, 123, 124]


@pytest.mark.parametrize("kernel,selection,copies", [(0, -1, 1), (1, 0, 1), (2, 3, 1), (3, 1, 1), (4, 2, 1), (5, 2, 1),
                                                     (-1, 2, 1), (5, 2, 360)])
def test_small_cells_rk4_matches_oracle(kernel, selection, copies):
    """copies = 360: more cells than the SMs hold CTAs of a warp per slot block (a warp
    per cell then); 70 steps on the first sizes cross the steps of one launch."""
    import torch

    rng = np.random.default_rng(70 + kernel)
    grids = [pg.grids.geometric_pow2(124, 1e-21, 4.0), make_grid("generic", 48, rng)]
    base_n = SIZES + [1, 31, 32, 48]
    base_g = [0] * len(SIZES) + [1] * 4
    N1 = [pg.grids.lognormal_ic(grids[g][:n], max(0, n // 4), 1.0, 1e12, cut=5.0) for g, n in zip(base_g, base_n)]
    k = [kk for kk in AGG_KERNELS if kk[0] == max(kernel, 0)][0]
    v_ref = np.array([grids[g][n // 2] for g, n in zip(base_g, base_n)])
    params = pg.batch.cell_params(len(base_n), beta0=1e-20, beta_br=k[2], beta_sh=k[3], S0=1e-3, v_ref=v_ref,
                                  alpha=1.2, v_min=v_ref)
    t_q, bw_q = pg.quadrature.uniform(4)
    dt = 0.5
    for steps in ((3,) if copies > 1 else (3, 70)):
        sel = slice(None) if steps == 3 else slice(0, 6)
        cn, cg = np.tile(base_n[sel], copies), np.tile(base_g[sel], copies)
        prm = np.tile(params[sel], (copies, 1))
        with pg.BatchPlan(grids, cn, cg, kernel, selection, t_q, bw_q) as plan:
            dN = t(np.concatenate(N1[sel] * copies))
            assert plan.rk4(dN, t(prm), dt, steps) == 0
            torch.cuda.synchronize()
            got = plan.split(dN.cpu().numpy())
        for c in range(len(N1[sel])):
            x, p = grids[cg[c]][:cn[c]], prm[c]
            agg = dict(kernel=kernel, beta0=p[0], beta_br=p[1], beta_sh=p[2]) if kernel >= 0 else None
            brk = (dict(t_q=t_q, bw_q=bw_q, selection=selection, S0=p[3], v_ref=p[4], alpha=p[5], v_min=p[6])
                   if selection >= 0 else None)
            ref = N1[c].copy()
            for _ in range(steps):
                ref = pyoracle.rk4_step(ref, x, dt, agg=agg, brk=brk)
            for r in range(copies):
                np.testing.assert_allclose(got[r * len(N1[sel]) + c], ref, rtol=1e-11, atol=1e-11 * np.abs(N1[c]).max(),
                                           err_msg="k=%d sel=%d n=%d copy %d" % (kernel, selection, cn[c], r))
