"""Spectra of a box so small that wavenumbers overflow single precision: modes off the axes have |k| =
infinity and land in the overflow bin, those with a zero component have infinity times zero, not
a number, and land in bin 0, as numpy.digitize would have it for each mode. Counts are exact."""

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from jfli_b200.power import poles_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (36, 24, 32), (64, 64, 64), (54, 16, 18)])
def test_infinite_wavenumbers(shape):
    m = torch.randn(*shape, device="cuda")
    edges = torch.tensor([0.1, 0.2, 0.5], device="cuda")
    on_axis = np.prod(shape) - np.prod([n - 1 for n in shape])
    want = [on_axis, 0, 0, np.prod(shape) - on_axis]
    counts = ops.power_sums(m, edges, (1e-38,) * 3)[1].cpu().numpy()
    assert counts.tolist() == want
    out, nell = poles_sums(m, None, (1e-38,) * 3, edges.cpu().numpy(), (0, 2), (0.0, 0.0, 1.0))
    assert out[0, 2 * nell].cpu().numpy().tolist() == want
