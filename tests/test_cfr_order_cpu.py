"""A path table out of canonical order is refused before anything else, also
where there is no GPU."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from witwin_channel_b200.channel import cfr


def test_unordered_host_table_is_refused():
    rx, v = torch.tensor([1, 0], dtype=torch.int32), torch.ones(2)
    table = SimpleNamespace(tx_id=torch.zeros_like(rx), rx_id=rx, delay_s=v, field_real=v, field_imag=v)
    with pytest.raises(ValueError, match="canonical"):
        cfr(table, np.arange(4) * 1e5, num_tx=1, num_rx=2)
