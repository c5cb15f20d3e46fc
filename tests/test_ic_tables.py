"""P(k) tables of the initial-condition filter whose points are spread in other ways than the usual
logarithmic one: linear from 0, two points, equal neighbours, the longest table, one that spans
many octaves beyond the mesh. Against the FP64 oracle, 1e-5 relative L2 as for the usual table."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

TABLES = {
    "linear": np.linspace(0.0, 2.5, 200),
    "two": np.array([1e-3, 4.0]),
    "repeated": np.sort(np.concatenate([np.logspace(-2, 0.6, 40), np.full(3, 0.2)])),
    "longest": np.concatenate([[0.0], np.logspace(-3, 0.6, 4095)]),
    "octaves": np.logspace(-30, 30, 500),
}


@pytest.mark.parametrize("name", TABLES)
@pytest.mark.parametrize("shape", [(16, 12, 8), (64, 32, 32), (18, 6, 18)])
def test_tables(name, shape):
    k = TABLES[name].astype(np.float32).astype(np.float64)
    pk = (1e3 / (1.0 + 3.0 * np.minimum(k, 8.0))).astype(np.float32).astype(np.float64)
    box = tuple(4.0 * n for n in shape)
    noise = np.random.default_rng(len(k)).standard_normal(shape).astype(np.float32)
    dev = lambda a: torch.as_tensor(np.asarray(a, np.float32), device="cuda")
    ic = ops.ic_filter(dev(noise), dev(k), dev(pk), box).cpu().numpy()
    assert rel_l2(ic, opm.ic_filter(noise.astype(np.float64), box, k, pk)) < 1e-5
