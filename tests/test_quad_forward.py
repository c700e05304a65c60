"""GPU test of the quad forward, whose rays keep a sample's far quad for the
next sample: it equals the register forward from 8-byte pairs at odd and tiny
sizes, for rays up and down the slices and along every axis.

Both take the same samples.  A sample may differ by its own roundings (at most
32 units of 2^-24 of the largest value, quads holding differences of
differences), by its position's (coordinates up to 4 n, four roundings, three
axes, slopes up to twice the largest value) and by the running sum's."""
import numpy as np
import pytest
import torch

from curadon_gb300 import ConeGeometry, forward
from curadon_gb300.phantom import cone_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tilt", [0.0, 0.4])
@pytest.mark.parametrize("shape,nangles,det", [((1, 1, 1), 8, (3, 5)), ((2, 7, 5), 12, (9, 33)),
                                               ((33, 9, 40), 16, (21, 70)),
                                               ((17, 40, 3), 7, (64, 31))])
def test_equals_register_forward(cuda_device, monkeypatch, shape, nangles, det, tilt):
    n = max(shape)
    g = cone_config(n, nangles, 1)
    g.update(vol_shape=shape, det_shape=det)
    if tilt:
        g["angles"] = np.stack([g["angles"], np.full_like(g["angles"], tilt),
                                np.full_like(g["angles"], -0.3)])
    x = torch.rand(shape, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(n))
    out = []
    for algo in ("quad", "alu"):
        monkeypatch.setenv("CURADON_GB300_ALGO", "fwd3d=" + algo)
        geom = ConeGeometry(**g)
        s = torch.zeros(geom.sinogram_shape(), device=cuda_device)
        forward(x, s, geom)
        out.append(s.double())
    samples = int(np.sqrt(sum((k + 2) ** 2 for k in shape))) + 3
    bound = 2.0 ** -24 * samples * (32 + samples + 96 * n)
    assert out[0].abs().max() > 0
    assert (out[0] - out[1]).abs().max() <= bound
