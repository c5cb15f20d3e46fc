"""The second-order LPT adjoint on non-cubic meshes and two sets at once: against the same call with
the x and z axes exchanged (FP32 transforms of another axis order, 1e-5 for potentials, three of
them in a row: 3e-5), and <lam, J v> = <J^T lam, v> with J v by central differences of the
map, which is quadratic in the field, so that they are exact up to FP32 rounding (1e-4)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

FACTORS = (0.7, -0.3, 0.9, 1.1)


@pytest.mark.parametrize("shape, batch", [((6, 8, 18), 1), ((16, 12, 8), 2), ((32, 18, 64), 1)])
def test_second_order(shape, batch):
    rng = np.random.default_rng(sum(shape))
    ic, v = (rng.standard_normal((batch, *shape)).astype(np.float32) for _ in range(2))
    lx, lv = (rng.standard_normal((batch, *shape, 3)).astype(np.float32) for _ in range(2))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    swap = lambda a: a.transpose(0, 3, 2, 1, *range(4, a.ndim))
    vec = lambda a: swap(a)[..., ::-1]
    got = ops.lpt_adjoint(dev(ic), 2, *FACTORS, dev(lx), dev(lv)).cpu().numpy()
    other = ops.lpt_adjoint(dev(swap(ic)), 2, *FACTORS, dev(vec(lx)), dev(vec(lv))).cpu().numpy()
    assert rel_l2(swap(other), got) < 3e-5
    lhs = 0.0
    for sign in (1.0, -1.0):
        dx, p = ops.lpt(dev(ic + np.float32(sign) * v), 2, *FACTORS)
        lhs += sign * 0.5 * float((dev(lx).double() * dx.double()).sum() + (dev(lv).double() * p.double()).sum())
    rhs = float((got.astype(np.float64) * v).sum())
    scale = np.linalg.norm(got.astype(np.float64)) * np.linalg.norm(v.astype(np.float64))
    assert abs(lhs - rhs) < 1e-4 * scale
