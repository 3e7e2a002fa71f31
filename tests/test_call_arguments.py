"""Arguments of the Python calls that need no tensor: raw device addresses and an
integer stream work where torch is not installed, and the current stream is found
with a torch that lacks the private shortcut to its handle."""
import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A child process: `stub` stands in for torch (None: importing it raises ImportError).
CHILD = """
import sys, types
sys.path.insert(0, %r)
class Block:
    def find_spec(self, name, path=None, target=None):
        if name.split(".")[0] == "torch":
            raise ModuleNotFoundError("No module named 'torch'")
sys.meta_path.insert(0, Block())
import pbe_gb300.rhs as r
""" % os.path.join(ROOT, "pbe-fixed-pivot-cuda_gb300")


def _child(code):
    out = subprocess.run([sys.executable, "-c", CHILD + textwrap.dedent(code)], capture_output=True,
                         text=True, timeout=120)
    assert out.returncode == 0, out.stderr[-1500:]


def test_addresses_and_streams_without_torch():
    _child("""
        assert r._ptr(4096, "N") == 4096 and r._ptr(0, "N") is None and r._ptr(None, "N") is None
        assert r._stream(77) == 77 and r._stream(0) is None
        assert r._stream(types.SimpleNamespace(cuda_stream=5)) == 5
        assert "torch" not in sys.modules
    """)


def test_call_on_addresses_without_torch():
    # the checks of the arguments run before any device is asked for
    _child("""
        from pbe_gb300 import AggregationParams, ERR_INVALID_DEVICE_POINTER
        p = AggregationParams(n=8, kernel_type=0, beta0=1.0)
        assert r.aggregation_rhs(4096, 0, 8192, p, stream=1) == ERR_INVALID_DEVICE_POINTER
    """)


@pytest.mark.parametrize("shortcut", [True, False])
def test_current_stream_handle(shortcut):
    _child("""
        t = types.ModuleType("torch")
        t.Tensor = type("Tensor", (), {})
        t._C = types.SimpleNamespace()
        if %r:
            t._C._cuda_getCurrentRawStream = lambda device: 40 + device
        t.cuda = types.SimpleNamespace(
            current_device=lambda: 3,
            current_stream=lambda device=None: types.SimpleNamespace(cuda_stream=43))
        sys.modules["torch"] = t
        assert r._stream(None) == 43
    """ % shortcut)
