"""Single instances small enough for one cluster of CTAs (up to 496 sections): every
number of CTAs up to the largest cluster, on grids whose work lies where it is hard to
share -- clipped pairs (fine and linear grids: up to half of all pairs), rows that end
early (linear), slots with many pairs beside slots with few (linear, then geometric).

Bound: the parity tests' 1e-12 of a bin's sum of |terms|; at the foot of a population
the same without a floor, down to 1e-290 (a product on the way to a bin is at most 1e-14
of its sum, and keeps 1e-13 of itself down to 5e-311)."""
import numpy as np
import pytest

import pbe_gb300 as pg
from gpu_util import AGG_KERNELS, agg_params, assert_close, dev, gpu_agg, make_grid, oracle_agg, t

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 31, 32, 62, 63, 93, 94, 155, 217, 248, 249, 280, 310, 311, 400, 434, 465, 495, 496, 497)


def linear_geometric(n):
    x = 1e-18 * np.arange(1, n + 1, dtype=np.float64)
    m = max(1, n // 2)
    x[m:] = x[m - 1] * 1.03 ** np.arange(1, n - m + 1)
    return x


GRIDS = {"q4": lambda n: pg.grids.geometric_pow2(n, 1e-21, 4.0),
         "q64": lambda n: pg.grids.geometric_pow2(n, 1e-21, 64.0),
         "q512": lambda n: pg.grids.geometric_pow2(n, 1e-21, 512.0),
         "linear": lambda n: make_grid("linear", n, None),
         "linear_geometric": linear_geometric,
         "irregular": lambda n: make_grid("generic", n, np.random.default_rng(n))}


def populations(x):
    n = len(x)
    i = np.arange(n)
    yield "smooth", 1e12 * np.exp(-0.5 * ((i - n / 3.0) / (n / 8.0 + 1.0)) ** 2)
    yield "holes", np.where(i % 2 == 0, 1e10, 0.0)
    N = 1e12 * np.exp(-0.5 * ((i - n // 3) / (n / 60.0 + 2.0)) ** 2)
    N[N < 1e-305] = 0.0
    yield "foot", N


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_small_instances_match_oracle(kernel, b0, bbr, bsh, grid):
    for n in SIZES:
        x = GRIDS[grid](n)
        p = agg_params(n, kernel, b0, bbr, bsh, x, geometric=grid.startswith("q"))
        for what, N in populations(x):
            ref, scale, _ = oracle_agg(N, x, p)
            code, got = gpu_agg(N, x, p, pg.MODE_GATHER)
            assert code == 0
            assert_close(got, ref, scale, "k=%d %s n=%d %s" % (kernel, grid, n, what))


@pytest.mark.parametrize("kernel,b0,bbr,bsh", AGG_KERNELS, ids=[str(k[0]) for k in AGG_KERNELS])
def test_small_instances_keep_a_populations_foot(kernel, b0, bbr, bsh):
    """As the window sums' test, for the cluster kernel's own prefix sums."""
    for n, q in ((200, 16.0), (300, 32.0), (480, 32.0)):
        x = pg.grids.geometric_pow2(n, 1e-21, q)
        p = agg_params(n, kernel, b0, bbr, bsh, x)
        for c, width in ((n // 4, 3.0), (n // 3, 2.0)):
            N = 1e12 * np.exp(-0.5 * ((np.arange(n) - c) / width) ** 2)
            N[N < 1e-305] = 0.0
            ref, scale, _ = oracle_agg(N, x, p)
            code, got = gpu_agg(N, x, p, pg.MODE_GATHER)
            assert code == 0
            foot = (scale > 1e-290) & (scale < 1e-200)
            assert foot.sum() >= 3
            err = np.abs(got - ref)[foot] / scale[foot]
            assert err.max() <= 1e-12, (kernel, n, c, err.max())


@pytest.mark.parametrize("n,grid", [(31, "linear"), (64, "q4"), (217, "linear"), (400, "q64"), (496, "linear_geometric"),
                                    (496, "irregular")])
def test_tape_stages_equal_the_calls(n, grid):
    """A tape's stages run on kept tables: bitwise RK4 of the drop-in calls."""
    import torch

    x = GRIDS[grid](n)
    N0 = 1e12 * np.exp(-0.5 * ((np.arange(n) - n / 3.0) / (n / 8.0 + 1.0)) ** 2)
    p = agg_params(n, 5, 0.0, 6.73e-18, 66.67)
    dt = 1e-9
    X, N = t(x), t(N0)

    def rhs(y):
        k = torch.zeros(n, dtype=torch.float64, device=dev())
        pg.check(pg.aggregation_rhs(y, X, k, p, mode=pg.MODE_GATHER))
        return k

    for _ in range(2):
        k1 = rhs(N)
        k2 = rhs(N + 0.5 * dt * k1)
        k3 = rhs(N + 0.5 * dt * k2)
        k4 = rhs(N + dt * k3)
        N = N + (dt / 6.0) * (((k1 + 2.0 * k2) + 2.0 * k3) + k4)
    tape = pg.Rk4Tape(2, dt, 1, [p])
    M = t(N0)
    pg.check(tape.forward(M, X))
    torch.cuda.synchronize()
    assert torch.equal(M, N)


def _median_us(fn, reps=31):
    import torch

    for _ in range(5):
        fn()
    ts = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        ts.append(a.elapsed_time(b) * 1e3)
    return float(np.median(ts))


def test_largest_clusters_keep_up_with_the_next_path():
    """480 sections at 128 an octave (most of their pairs direct or clipped) took twice as
    long by the cluster as 520 by the path above it while one CTA summed all clipped
    pairs; 1.3 times since."""
    import torch

    us = []
    for n in (480, 520):
        x = pg.grids.geometric_pow2(n, 1e-21, 128.0)
        N, X = t(1e12 * np.exp(-0.5 * ((np.arange(n) - n / 3.0) / 60.0) ** 2)), t(x)
        rhs = torch.zeros(n, dtype=torch.float64, device=dev())
        p = agg_params(n, 5, 0.0, 6.73e-18, 66.67, x)
        us.append(_median_us(lambda: pg.aggregation_rhs(N, X, rhs, p, mode=pg.MODE_GATHER)))
    assert us[0] <= 1.65 * us[1], us
