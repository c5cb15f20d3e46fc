"""A call whose tables (FFT twiddles, HEALPix rings) are first needed while a stream is captured: the
mixed 2^a 3^b lengths, which other calls have not met. In a process of its own, where no test
has made the tables. The replay runs the kernels of the plain call: the same bits from the
transforms; the shells' atomics add in any order (1e-5 of the largest value)."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

SCRIPT = """
import torch
from jfli_b200 import ops
torch.manual_seed(1)
m = torch.randn(36, 54, 144, device="cuda")
x = torch.randn(16, 16, 16, 3, device="cuda")
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode="{mode}"):
    spec = ops.rfft3d(m)
    back = ops.irfft3d(spec, 144)
    shells = ops.healpix_paint(x, 32, (64.0,) * 3, (31.0,) * 3, 2.0, 30.0)
g.replay()
torch.cuda.synchronize()
assert torch.equal(spec, ops.rfft3d(m)) and torch.equal(back, ops.irfft3d(spec, 144))
want = ops.healpix_paint(x, 32, (64.0,) * 3, (31.0,) * 3, 2.0, 30.0)
assert float((shells - want).abs().max()) <= 1e-5 * float(want.max()) and float(want.sum()) > 100.0
assert float((back - m).abs().max()) < 1e-5
"""


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_tables_first_needed_in_a_capture(mode):
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(mode=mode)], capture_output=True, text=True, timeout=300,
                         cwd=Path(__file__).resolve().parents[1])
    assert run.returncode == 0, run.stderr[-1500:]
