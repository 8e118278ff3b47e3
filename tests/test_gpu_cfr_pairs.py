"""The paired CFR kernel (even grids of more than 256 subcarriers, an even
count) at the edges of its passes, and the odd counts and short spectra beside
it that keep the scalar kernel, against the defining sum in FP64.

Tolerance: a start phasor and a step are each within 4e-7 (argument reduced in
FP64, hardware sine), the step is applied at most 16 times, and the rotation
rounds 16 times by 2^-23: below 1e-5 of the link's sum of path magnitudes.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from witwin_channel_b200.channel import cfr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subcarriers", [2, 256, 257, 258, 511, 512, 514, 1023, 1024, 1026, 2050])
@pytest.mark.parametrize("normalize", [True, False])
def test_even_grid_equals_defining_sum(subcarriers, normalize):
    links, rng = 9, np.random.default_rng(subcarriers)
    count = np.array([0, 1, 2, 40, 3, 0, 1, 33, 5])
    rx = np.repeat(np.arange(links), count)
    n = rx.size
    delay = (1e-7 + rng.exponential(2e-7, n)).astype(np.float32)
    re, im = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    dev = "cuda"
    table = SimpleNamespace(tx_id=torch.zeros(n, dtype=torch.int32, device=dev),
                            rx_id=torch.tensor(rx, dtype=torch.int32, device=dev),
                            delay_s=torch.tensor(delay, device=dev), field_real=torch.tensor(re, device=dev),
                            field_imag=torch.tensor(im, device=dev))
    freqs = (np.arange(subcarriers) - subcarriers // 2) * 390.625e3
    got = cfr(table, freqs, num_tx=1, num_rx=links, normalize_delays=normalize)[0].cpu().numpy()
    for link in range(links):
        own = rx == link
        tau = delay[own].astype(np.float64)
        if normalize and tau.size:
            tau = tau - tau.min()
        a = re[own].astype(np.float64) + 1j * im[own]
        want = (a[:, None] * np.exp(-2j * math.pi * tau[:, None] * freqs[None])).sum(0)
        assert np.abs(got[link] - want).max() <= 1e-5 * np.abs(a).sum()


def test_unordered_table_is_refused():
    t = torch.tensor([1, 0], dtype=torch.int32, device="cuda")
    v = torch.ones(2, device="cuda")
    table = SimpleNamespace(tx_id=torch.zeros_like(t), rx_id=t, delay_s=v, field_real=v, field_imag=v)
    with pytest.raises(ValueError):
        cfr(table, np.arange(300) * 1e5, num_tx=1, num_rx=2)
