"""A call that fails (here: on a stream whose capture has been invalidated, an error of
the host's making) returns its error, and the next call succeeds: no error stays behind."""
import contextlib
import ctypes

import numpy as np
import pytest

import pbe_gb300 as pg
from gpu_util import agg_params, dev, t

pytestmark = pytest.mark.gpu


def _cudart():
    import torch

    torch.zeros(1, device=dev())
    with open("/proc/self/maps") as f:
        libs = {line.split()[-1] for line in f if "libcudart" in line}
    if not libs:
        pytest.skip("no shared CUDA runtime in this process")
    return ctypes.CDLL(sorted(libs)[0])


@contextlib.contextmanager
def broken_stream():
    rt = _cudart()
    s = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    assert rt.cudaStreamBeginCapture(s, 2) == 0              # relaxed: no other thread is held up
    assert rt.cudaStreamSynchronize(s) != 0                  # not allowed while capturing: invalidates it
    rt.cudaGetLastError()
    yield s.value
    g = ctypes.c_void_p()
    rt.cudaStreamEndCapture(s, ctypes.byref(g))
    rt.cudaGetLastError()
    assert rt.cudaStreamDestroy(s) == 0


def _cells():
    x = pg.grids.geometric_pow2(60, 1e-21, 4.0)
    plan = pg.BatchPlan([x], [60, 40], [0, 0], 5)
    N = t(np.concatenate([np.exp(-0.5 * (np.arange(n) - 20.0) ** 2 / 25.0) * 1e12 for n in (60, 40)]))
    return plan, N, t(pg.batch.cell_params(2, beta_br=6.73e-18, beta_sh=66.67))


@pytest.mark.parametrize("call", ["rhs", "vjp", "jvp"])
def test_batch_calls_leave_no_error_behind(call):
    import torch

    plan, N, prm = _cells()
    out, gp = torch.zeros_like(N), torch.zeros(2, 8, dtype=torch.float64, device=dev())
    calls = {"rhs": lambda s: plan.rhs(N, out, prm, stream=s),
             "vjp": lambda s: plan.rhs_vjp(N, N, out, gp, prm, stream=s),
             "jvp": lambda s: plan.jvp(N, N, out, prm, stream=s)}
    assert calls[call](None) == 0                            # what is set up on the first call
    with broken_stream() as s:
        assert calls[call](s) != 0
    assert calls[call](None) == 0
    torch.cuda.synchronize()
    plan.close()


def test_small_instance_leaves_no_error_behind():
    import torch

    n = 64
    x = t(pg.grids.geometric_pow2(n, 1e-21, 4.0))
    N, rhs = t(np.ones(n)), torch.zeros(n, dtype=torch.float64, device=dev())
    p = agg_params(n, 5, 0.0, 6.73e-18, 66.67)
    ws = torch.zeros(pg.aggregation_workspace_bytes(n), dtype=torch.uint8, device=dev())
    assert pg.aggregation_rhs(N, x, rhs, p, workspace=ws) == 0
    with broken_stream() as s:
        assert pg.aggregation_rhs(N, x, rhs, p, stream=s, workspace=ws) != 0
    assert pg.aggregation_rhs(N, x, rhs, p, workspace=ws) == 0
    torch.cuda.synchronize()
