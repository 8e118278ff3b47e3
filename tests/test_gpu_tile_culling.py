"""Tile-level rejection changes no path: the reflection and diffraction kernels
drop a candidate for a whole 32-receiver tile when the tile's bounds prove
that no receiver can have it (back projection outside a group's box, or one
triangle across the whole shaft).  The same receivers in shuffled order, among
as many others over the whole scene as it takes to pass the 2,048 pairs up to
which each point has a tile of its own, fill their tiles with far-apart points,
whose bounds span the scene and reject next to nothing: both must give the
same rows bit for bit.  The sizes take each number of warps per tile (8 below
1,024 tiles, 4 below 4,096, then 2; the UTD kernel 8, 4 and 2 from 4,096 and
16,384; FP64 always 8), with ragged edges; the scenes are boxes, subdivided
roofs and glass sheets, far from the origin, under several transmitters whose
tiles share blocks, and on tilted and upright receiver planes, whose tiles are
boxes and not flat."""

from __future__ import annotations

import pytest
import torch

from witwin_channel_b200 import _native, engine
from witwin_channel_b200.compiler import compile_scene, receiver_setup
from witwin_channel_b200.deterministic import _endpoints
from witwin_channel_b200.scene import Scene, make_receiver_grid, make_transmitter
from witwin_channel_b200.workloads import city_layout, city_scene

pytestmark = pytest.mark.gpu

FLAT = ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0))


def _rows(compiled, ep, mats, depth, rx_of, components, precision):
    """The solve's path records as sorted integer keys, the length's bits last;
    records of receivers that map to -1 left out."""
    rows = engine.run_solve(compiled, ep, mats, [28e9], components=engine.component_bits(components), max_depth=depth,
                            coherent=True, want_rows=True, precision=precision)["rows"]
    dec = engine.decode_rows(rows, engine.select_rows(rows, depth, None, "global"))
    key = torch.stack([rx_of[dec["rx_id"].long()], dec["tx_id"].long(), dec["component_id"].long(),
                       dec["depth"].long(), dec["edge_id"].long(), *dec["seq"].long().unbind(1),
                       dec["length"].view(torch.int32).long()], 1)
    key = key[key[:, 0] >= 0]
    order = torch.arange(key.shape[0], device=key.device)
    for c in range(key.shape[1] - 1, -1, -1):
        order = order[torch.sort(key[order, c], stable=True).indices]
    return key[order]


def _check(rows, cols, boxes, depth, spacing, *, axes=FLAT, origin_z=1.5, offset=(0.0, 0.0, 0.0), txs=1, glass=False,
           precision=_native.PRECISION_MIXED):
    layout = city_layout(boxes, 11)
    shift = torch.tensor(offset)
    sheets = [((0.5 * (x0 + x1), y0 + 0.5), (0.5 * (x0 + x1), y1 - 0.5), 0.8 * h) for x0, y0, x1, y1, h in layout.boxes[::3]]
    structures = city_scene(layout, roof_k=(lambda b: 3 if b % 2 else 4) if glass else None, sheets=sheets if glass else None)
    for st in structures:
        st.geometry.vertices = st.vertices + shift
    spots = [(layout.lot_size - layout.half, 3.0, 27.0), (2.0, layout.lot_size - layout.half, 8.0),
             (layout.lot_size - layout.half, -40.0, 75.0)][:txs]
    transmitters = [make_transmitter(tuple(float(a + b) for a, b in zip(p, offset))) for p in spots]
    x, y = (torch.tensor(a) for a in axes)
    origin = torch.tensor([0.0, 0.0, origin_z]) + shift - x * ((rows - 1) / 2 * spacing)
    origin = origin - torch.tensor([1.0, 1.0, 0.0]) * y * ((cols - 1) / 2 * spacing)
    grid = make_receiver_grid(origin=tuple(origin.tolist()), x_axis=axes[0], y_axis=axes[1], shape=(rows, cols),
                              spacing=(spacing, spacing))
    scene = Scene(structures=structures, endpoints=[*transmitters, grid])
    device = torch.device("cuda", torch.cuda.current_device())
    compiled = compile_scene(scene, device)
    mats = compiled.material_tables([28e9], device)
    ep = _endpoints(scene, device)
    n = rows * cols
    g = torch.Generator().manual_seed(5)
    others = max(0, 4096 - n)
    span = torch.tensor([2.0 * layout.half, 2.0 * layout.half, 60.0])
    spread = (torch.rand((others, 3), generator=g) - torch.tensor([0.5, 0.5, 0.0])) * span + shift
    positions = torch.cat([grid.points().to(device), spread.to(device)])
    ids = torch.cat([torch.arange(n), torch.full((others,), -1)])
    perm = torch.randperm(n + others, generator=g)
    pol = receiver_setup(scene, device)["pol"].reshape(-1, 3)[:1].expand(n + others, 3).contiguous()
    points = {"kind": "point", "grid": None, "count": n + others, "shape": None, "pol": pol, "pol_stride": 3,
              "positions": positions[perm.to(device)].contiguous()}
    shuffled = engine.Endpoints(tx_pos=ep.tx_pos, tx_power=ep.tx_power, tx_pol=ep.tx_pol, rx=points)
    components = {"los", "reflection", "diffraction"} | ({"transmission"} if glass else set())
    a = _rows(compiled, ep, mats, depth, torch.arange(n, device=device), components, precision)
    b = _rows(compiled, shuffled, mats, depth, ids[perm].to(device), components, precision)
    assert a.shape[0] > 0
    assert torch.equal(a, b)


@pytest.mark.parametrize("rows,cols,boxes,depth,spacing", [
    (1, 1, 12, 2, 2.0),        # one receiver
    (37, 29, 16, 3, 4.1),      # 8 warps per tile, ragged in both directions
    (189, 181, 40, 2, 1.9),    # 4 warps per tile
    (403, 397, 12, 1, 0.5),    # 2 warps per tile, the UTD kernel 4
    (733, 719, 9, 1, 0.21),    # 2 warps per tile in both
])
def test_grid_rows_equal_shuffled_points(rows, cols, boxes, depth, spacing):
    _check(rows, cols, boxes, depth, spacing)


@pytest.mark.parametrize("shape", [(45, 61), (189, 181)])  # 8 and 4 warps per tile
@pytest.mark.parametrize("options", [
    {"glass": True},
    {"offset": (1.0e4, -7.3e3, 40.0)},
    {"axes": ((1.0, 0.0, 0.0), (0.0, 0.6, 0.8)), "origin_z": 2.0},   # tilted
    {"axes": ((0.8, 0.6, 0.0), (0.0, 0.0, 1.0)), "origin_z": 0.7},   # upright, across the streets
    {"glass": True, "axes": ((0.8, 0.0, 0.6), (0.0, 1.0, 0.0)), "offset": (2.0e3, 1.0e3, 0.0)},
], ids=["glass", "far", "tilted", "upright", "tilted-glass"])
def test_scenes_and_planes(shape, options):
    _check(*shape, 16, 2, 1.3, **options)


def test_transmitters_share_blocks():
    _check(152, 76, 16, 2, 2.1, txs=3)  # 361 tiles each, 1,083 in all: two to a block


@pytest.mark.parametrize("options", [{}, {"glass": True, "txs": 3}, {"axes": ((1.0, 0.0, 0.0), (0.0, 0.6, 0.8))}],
                         ids=["flat", "glass", "tilted"])
def test_fp64(options):
    _check(45, 61, 16, 2, 1.3, precision=_native.PRECISION_FP64, **options)
