"""More small maps at once than a launch's grid takes: every map's a_lm is that of the map alone (the
same kernels in the same order: the same bits)."""

import pytest
import torch

from jfli_b200 import sht

pytestmark = pytest.mark.gpu


def test_more_maps_than_one_launch_takes():
    maps = torch.randn(65600, 12, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    alms = sht.maps2alm(maps, 2, iter=1)
    assert len(alms) == len(maps)
    for i in (0, 1, 65534, 65535, 65599):
        assert torch.equal(alms[i], sht.map2alm(maps[i], 2, iter=1))
