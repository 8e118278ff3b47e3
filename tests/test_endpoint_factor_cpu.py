"""Array weights of many endpoints in batches equal the weights of one endpoint
at a time: every pattern kind, turned and unturned arrays, a custom pattern and
an object that stands for several endpoints.  Tolerance: phases up to 13 rad as
FP32 sums of three products in another order, 3 x 2^-24 x 13 each way."""

from __future__ import annotations

import pytest
import torch

from witwin_channel_b200 import path
from witwin_channel_b200.scene import AntennaPattern, make_receiver

C0 = 299_792_458.0


def _endpoint(g, pattern, turned):
    kw = {"orientation": torch.rand(3, generator=g) * 2.0} if turned else {}
    return make_receiver(torch.rand(3, generator=g), pattern=pattern,
                         element_positions=(torch.rand((3, 3), generator=g) - 0.5) * 0.05, **kw)


@pytest.mark.parametrize("conjugate", [False, True])
@pytest.mark.parametrize("kinds", [("isotropic",), ("vertical", "horizontal", "isotropic", "custom")])
@pytest.mark.parametrize("turned", [False, True])
def test_batched_weights_equal_single_endpoints(kinds, turned, conjugate):
    g = torch.Generator().manual_seed(len(kinds) + 2 * turned)
    custom = AntennaPattern("custom", lambda d: (d[..., 0] + 1j * d[..., 2]).to(torch.complex64))
    endpoints = [_endpoint(g, custom if k == "custom" else k, turned and i % 2 == 0)
                 for i, k in enumerate(kinds * 3)]
    shared = _endpoint(g, "isotropic", turned)
    endpoints[1:1] = [shared, shared]
    directions = torch.randn((len(endpoints), 2, 5, 3), generator=g)
    f = 8.0e9
    got = path._endpoint_factor(endpoints, directions, frequency_hz=f, conjugate_pattern=conjugate)
    for i, e in enumerate(endpoints):
        pattern = path.pattern_field_response(e.pattern, path._local_direction(directions[i], e))
        if conjugate:
            pattern = pattern.conj()
        want = path.steering_vector(e, directions[i], frequency_hz=f) * pattern.unsqueeze(-1)
        torch.testing.assert_close(got[i], want, rtol=1e-5, atol=1e-5)
