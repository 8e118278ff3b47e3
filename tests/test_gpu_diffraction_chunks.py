"""Edge chunks of several transmitters whose edge lists differ in length.  From
4,096 tiles a block of the UTD kernel holds two tiles, and with an odd tile
count per transmitter one block holds the last tile of one transmitter and the
first of the next; in a chunk past the first one's edges only the second's
half has work.

Tolerance: one chunk and many sum the same terms per cell; splitting the sum
into partial FP32 sums moves each by a few 2^-24 of the terms' magnitudes:
1e-5 of the value, and 1e-6 of the map's largest value where terms cancel."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from witwin_channel_b200 import _native, engine
from witwin_channel_b200.compiler import compile_scene
from witwin_channel_b200.deterministic import _endpoints
from witwin_channel_b200.scene import Scene, make_receiver_grid, make_transmitter
from witwin_channel_b200.workloads import city_layout, city_scene, street_point

pytestmark = pytest.mark.gpu


def _solve(structures, transmitters, grid, freqs):
    scene = Scene(structures=structures, endpoints=[*transmitters, grid])
    device = torch.device("cuda", torch.cuda.current_device())
    compiled = compile_scene(scene, device)
    ep = _endpoints(scene, device)
    cells = engine.alloc_cells(len(freqs), ep.num_tx, ep.num_rx, device)
    engine.run_solve(compiled, ep, compiled.material_tables(freqs, device), freqs,
                     components=engine.component_bits({"diffraction"}), max_depth=1, coherent=True, cells=cells)
    return cells


def _edges_kept(structures, transmitter, freqs):
    """Edges that the solve keeps for one transmitter."""
    grid = make_receiver_grid(origin=(0.0, 0.0, 1.5), x_axis=(1.0, 0.0, 0.0), y_axis=(0.0, 1.0, 0.0), shape=(1, 1),
                              spacing=(1.0, 1.0))
    _native.profile_enable(True)
    try:
        _solve(structures, [transmitter], grid, freqs)
        return _native.profile_read()["edges"]
    finally:
        _native.profile_enable(False)


@pytest.mark.parametrize("freqs", [[28e9], [3.5e9, 6e9, 28e9, 39e9, 60e9]])
def test_chunks_of_unequal_transmitters_match_one_chunk(monkeypatch, freqs):
    layout = city_layout(20, 3, lot_size=30.0, footprint=(8.0, 20.0), height=(6.0, 25.0))
    structures = city_scene(layout)
    rng = np.random.default_rng(3)
    txs = [make_transmitter(street_point(layout, rng, z)) for z in (1.2, 40.0, 9.0)]
    kept = [_edges_kept(structures, t, freqs) for t in txs]
    assert -(-kept[0] // 32) < -(-kept[1] // 32), kept  # the first one's edges end in an earlier chunk of 32
    rows, cols = 27 * 8, 51 * 4  # 1,377 tiles of 8 x 4 cells per transmitter, 4,131 in all
    grid = make_receiver_grid(origin=(-(rows - 1) / 2 * 0.7, -(cols - 1) / 2 * 0.7, 1.5), x_axis=(1.0, 0.0, 0.0),
                              y_axis=(0.0, 1.0, 0.0), shape=(rows, cols), spacing=(0.7, 0.7))
    one = _solve(structures, txs, grid, freqs)
    monkeypatch.setenv("WCB_DIFFRACTION_CHUNK_WORDS", "1")
    many = _solve(structures, txs, grid, freqs)
    for a, b in ((one.comp_power[2], many.comp_power[2]), (one.diff_vec_power, many.diff_vec_power),
                 (one.path_gain, many.path_gain)):
        a, b = a.double(), b.double()
        assert all(float(a[:, t].max()) > 0 for t in range(len(txs)))
        assert torch.all((a - b).abs() <= 1e-5 * a.abs() + 1e-6 * float(a.abs().max()))
