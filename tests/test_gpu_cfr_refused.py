"""A path table out of canonical order is refused without computing its
spectrum: the kernels test the check's device byte and leave the output as it
was.  Links of a permuted table span almost every record, so its spectrum
would cost links x records x subcarriers."""

from __future__ import annotations

import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from witwin_channel_b200 import _native
from witwin_channel_b200.channel import cfr

pytestmark = pytest.mark.gpu

LINKS, PER_LINK = 70, 3


def _table(order):
    rx = torch.arange(LINKS, dtype=torch.int32).repeat_interleave(PER_LINK)[order].cuda()
    g = torch.Generator().manual_seed(1)
    delay, re, im = (torch.rand(rx.numel(), generator=g).cuda() for _ in range(3))
    return SimpleNamespace(tx_id=torch.zeros_like(rx), rx_id=rx, delay_s=delay * 1e-6, field_real=re, field_imag=im)


@pytest.mark.parametrize("subcarriers", [7, 300, 511])  # one pass, paired lanes, an odd count
@pytest.mark.parametrize("even", [True, False])
def test_refused_call_leaves_the_output(subcarriers, even):
    t = _table(torch.arange(LINKS * PER_LINK))
    a = torch.view_as_real(torch.complex(t.field_real, t.field_imag).contiguous())
    freqs = torch.arange(subcarriers, dtype=torch.float64, device="cuda") * 1e5
    if not even:
        freqs[-1] += 3e4
    lib = _native.load()
    nbytes = ctypes.c_int64()
    _native.check(lib.wcb_cfr_workspace_size(1, LINKS, ctypes.byref(nbytes)), "wcb_cfr_workspace_size")
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device="cuda")
    outs = {}
    for refuse in (None, False, True):
        flag = None if refuse is None else torch.tensor(refuse, device="cuda")
        out = torch.full((1, LINKS, subcarriers), 7.0, dtype=torch.complex64, device="cuda")
        _native.check(lib.wcb_cfr_guarded(
            t.tx_id.data_ptr(), t.rx_id.data_ptr(), t.delay_s.data_ptr(), a.data_ptr(), t.rx_id.numel(), 1, LINKS,
            subcarriers, 0.0, 1e5 if even else 0.0, None if even else freqs.data_ptr(), 1, _native.ptr(flag),
            out.data_ptr(), ws.data_ptr(), ws.numel(), _native.stream_handle(out.device)), "wcb_cfr_guarded")
        outs[refuse] = out.cpu()
    assert torch.equal(outs[None], outs[False])
    assert not torch.any(outs[False] == 7.0)
    assert torch.all(outs[True] == 7.0)


@pytest.mark.parametrize("stream", [False, True])
def test_permuted_table_is_refused(stream):
    order = torch.randperm(LINKS * PER_LINK, generator=torch.Generator().manual_seed(2))
    with torch.cuda.stream(torch.cuda.Stream() if stream else torch.cuda.current_stream()):
        t = _table(order)
        with pytest.raises(ValueError, match="canonical"):
            cfr(t, np.arange(300) * 1e5, num_tx=1, num_rx=LINKS)


def test_check_is_read_after_its_own_copy(monkeypatch):
    """The event that the host waits for is recorded on the stream that holds
    the check's copy: the table's device, whatever the current device is."""
    streams = []

    class Event(torch.cuda.Event):
        def record(self, stream=None):
            streams.append(stream)
            super().record(stream)

    monkeypatch.setattr(torch.cuda, "Event", Event)
    t = _table(torch.arange(LINKS * PER_LINK))
    cfr(t, np.arange(300) * 1e5, num_tx=1, num_rx=LINKS)
    assert [s.cuda_stream for s in streams] == [_native.stream_handle(t.rx_id.device)]
    assert streams[0].device == t.rx_id.device
