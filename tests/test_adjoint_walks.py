"""The column walks of the reverse sweep's cotangent paint and divergence (meshes with ny a multiple
of 8 and nz of 32: equal ranges up to 2^22 cells, slabs above; the divergence by columns from 2^19
cells) against the same step with the x and z axes exchanged, which takes the grid-stride walk
and the stencil. Few planes per CTA, pieces that end inside a column, a last slab that is not
full, two particle sets, arrays that are not 16-byte aligned. One step: FP32 transforms of
another axis order, 1e-5 for potentials, so 2e-5 for what is read out of them."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _device(a, offset):
    flat = torch.empty(a.size + offset, dtype=torch.float32, device="cuda")[offset:]
    flat.copy_(torch.as_tensor(a.reshape(-1)))
    return flat.view(a.shape)


@pytest.mark.parametrize("shape, batch, offset", [((6, 8, 32), 1, 0), ((18, 16, 64), 2, 0), ((18, 16, 64), 1, 1),
                                                  ((36, 64, 256), 1, 0), ((18, 512, 512), 1, 0)])
def test_reverse_step_against_exchanged_axes(shape, batch, offset):
    rng = np.random.default_rng(sum(shape) + batch)
    fields = [s * rng.standard_normal((batch, *shape, 3)).astype(np.float32) for s in (np.float32(1.5), 1, 1, 1)]
    fields[1] *= np.float32(0.2)
    swap = lambda a: np.ascontiguousarray(a.transpose(0, 3, 2, 1, 4)[..., ::-1])
    out = []
    for f in (lambda a: a, swap):
        x, v, lx, lv = (_device(f(a), offset) for a in fields)
        sens = ops.kkd_adjoint(x, v, lx, lv, [0.3], [0.4])
        out.append([f(t.cpu().numpy()) for t in (x, v, lx, lv)] + [sens.cpu().numpy()])
    for a, b in zip(*out):
        assert rel_l2(a, b) < 2e-5
