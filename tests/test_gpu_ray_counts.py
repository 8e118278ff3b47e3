"""Rays answered and rays traced.  The diffraction visibility kernel searches
each (tile, edge) pair once; a pair that one triangle closes answers a query of
each of its cells without a trace, and an open pair traces one or two segments
per cell.  Tiles without a ragged edge hold 32 cells."""

from __future__ import annotations

import pytest

from tests import scenes
from witwin_channel_b200 import Config, _native, solve

pytestmark = pytest.mark.gpu


def _profile(components):
    scene, freq = scenes.small_city(n_boxes=16, seed=5, grid=(48, 40), spacing=2.0)
    _native.profile_enable(True)
    try:
        solve(scene, Config(components=components, max_depth=1), reference_frequency_hz=freq)
        return _native.profile_read()
    finally:
        _native.profile_enable(False)


def test_traced_rays_leave_out_the_cells_of_hidden_pairs():
    prof = _profile({"los", "diffraction"})
    pairs = (48 // 8) * (40 // 4) * prof["edges"]
    assert pairs > 0
    segments = prof["kernel_rays_traced"]["k_diffract"] - pairs
    hidden = prof["kernel_rays"]["k_diffract"] - segments
    assert hidden % 32 == 0 and 0 < hidden // 32 < pairs
    open_pairs = pairs - hidden // 32
    assert 32 * open_pairs <= segments <= 64 * open_pairs
    assert prof["kernel_rays_traced"]["k_los_trans"] == 48 * 40
    assert prof["rays_traced"] == sum(prof["kernel_rays_traced"].values())
    assert prof["acc_rays_traced"] == prof["rays_traced"] + prof["prep_rays"]


def test_other_kernels_trace_what_they_answer():
    prof = _profile({"los", "reflection"})
    assert prof["kernel_rays_traced"]["k_reflect"] == prof["kernel_rays"]["k_reflect"] > 0
    assert prof["rays_traced"] == prof["rays"] and prof["acc_rays_traced"] == prof["acc_rays"]
