"""sfsim_atmo_build_static as the only call of a process: it must not need what
other builds create (streams, events, an arena), on the legacy default stream
or another.  Afterwards the same process builds the tables by
sfsim_atmo_build_device, which the static ones equal bit for bit."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, sys
import torch
from sfsim_gb300 import _lib, atmosphere_lut as A, config as C
L = _lib.load()
cfg = C.small_fp64(precision=int(sys.argv[2]))
stream = torch.cuda.Stream() if sys.argv[1] == "created" else torch.cuda.default_stream()
def build(fn):
    out = [torch.full(s, -1.0, device="cuda") for s in A.table_shapes(cfg)]
    torch.cuda.synchronize()
    _lib.check(fn(ctypes.byref(cfg), *[t.data_ptr() for t in out], ctypes.c_void_p(stream.cuda_stream)), fn.__name__)
    torch.cuda.synchronize()
    return out
static = build(L.sfsim_atmo_build_static)
for a, b in zip(static, build(L.sfsim_atmo_build_device)):
    assert torch.isfinite(a).all() and torch.equal(a, b)
"""


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("stream", ["default", "created"])
def test_static_build_first(stream, precision):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", PROGRAM, stream, str(precision)], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
