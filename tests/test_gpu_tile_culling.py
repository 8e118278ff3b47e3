"""Tile-level rejection changes no path: the reflection and diffraction kernels
drop a candidate for a whole 32-receiver tile when the tile's bounds prove
that no receiver can have it (back projection outside a group's box, or one
triangle across the whole shaft).  The same receivers in shuffled order fill
their tiles with far-apart points, whose bounds span the scene and reject
next to nothing, so both orders must give the same rows bit for bit.  The
sizes take each number of warps per tile (8 below 1,024 tiles, 4 below 4,096,
then 2; the UTD kernel 8, 4 and 2 from 4,096 and 16,384), with ragged edges."""

from __future__ import annotations

import pytest
import torch

from witwin_channel_b200 import engine
from witwin_channel_b200.compiler import compile_scene, receiver_setup
from witwin_channel_b200.deterministic import _endpoints
from witwin_channel_b200.scene import Scene, make_receiver_grid, make_transmitter
from witwin_channel_b200.workloads import city_layout, city_scene

pytestmark = pytest.mark.gpu


def _rows(compiled, ep, mats, depth, rx_of):
    """The solve's path records as sorted integer keys, the length's bits last."""
    bits = engine.component_bits({"los", "reflection", "diffraction"})
    rows = engine.run_solve(compiled, ep, mats, [28e9], components=bits, max_depth=depth, coherent=True,
                            want_rows=True)["rows"]
    dec = engine.decode_rows(rows, engine.select_rows(rows, depth, None, "global"))
    key = torch.stack([rx_of[dec["rx_id"].long()], dec["component_id"].long(), dec["depth"].long(),
                       dec["edge_id"].long(), *dec["seq"].long().unbind(1),
                       dec["length"].view(torch.int32).long()], 1)
    order = torch.arange(key.shape[0], device=key.device)
    for c in range(key.shape[1] - 1, -1, -1):
        order = order[torch.sort(key[order, c], stable=True).indices]
    return key[order]


@pytest.mark.parametrize("rows,cols,boxes,depth,spacing", [
    (1, 1, 12, 2, 2.0),        # one receiver
    (37, 29, 16, 3, 4.1),      # 8 warps per tile, ragged in both directions
    (189, 181, 40, 2, 1.9),    # 4 warps per tile
    (403, 397, 12, 1, 0.5),    # 2 warps per tile, the UTD kernel 4
    (733, 719, 9, 1, 0.21),    # 2 warps per tile in both
])
def test_grid_rows_equal_shuffled_points(rows, cols, boxes, depth, spacing):
    layout = city_layout(boxes, 11)
    tx = make_transmitter((layout.lot_size - layout.half, 3.0, 27.0))
    grid = make_receiver_grid(origin=(-(rows - 1) / 2 * spacing, -(cols - 1) / 2 * spacing, 1.5), x_axis=(1.0, 0.0, 0.0),
                              y_axis=(0.0, 1.0, 0.0), shape=(rows, cols), spacing=(spacing, spacing))
    scene = Scene(structures=city_scene(layout), endpoints=[tx, grid])
    device = torch.device("cuda", torch.cuda.current_device())
    compiled = compile_scene(scene, device)
    mats = compiled.material_tables([28e9], device)
    ep = _endpoints(scene, device)
    n = rows * cols
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(5)).to(device)
    pol = receiver_setup(scene, device)["pol"].expand(n, 3).contiguous()
    points = {"kind": "point", "grid": None, "count": n, "shape": None, "pol": pol, "pol_stride": 3,
              "positions": grid.points().to(device)[perm].contiguous()}
    shuffled = engine.Endpoints(tx_pos=ep.tx_pos, tx_power=ep.tx_power, tx_pol=ep.tx_pol, rx=points)
    a = _rows(compiled, ep, mats, depth, torch.arange(n, device=device))
    b = _rows(compiled, shuffled, mats, depth, perm)
    assert a.shape[0] > 0
    assert torch.equal(a, b)
