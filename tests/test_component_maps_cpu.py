"""Component maps of a grid: the layout (T, cols, rows) of every slot, each in a
storage of its own, so a program that keeps or saves one map keeps that one."""

from __future__ import annotations

import pytest
import torch

from witwin_channel_b200.deterministic import _layout, _layout_slots


@pytest.mark.parametrize("transmitters", [0, 1, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.complex64])
def test_grid_maps_have_their_own_storage(transmitters, dtype):
    slots, shape = 3, (5, 7)
    rx = {"kind": "grid", "shape": shape}
    cells = torch.randn((slots, transmitters, shape[0] * shape[1]), dtype=dtype)
    maps = _layout_slots(cells, rx)
    assert len(maps) == slots
    for k, m in enumerate(maps):
        assert torch.equal(m, _layout(cells[k], rx))
        assert m.is_contiguous() and m.shape == (transmitters, shape[1], shape[0])
        assert m.untyped_storage().nbytes() == m.numel() * m.element_size()


def test_point_maps():
    cells = torch.randn((3, 2, 11))
    for k, m in enumerate(_layout_slots(cells, {"kind": "point"})):
        assert torch.equal(m, cells[k])
