"""GPU test of the matched adjoints' merged atomics: the adjoint equals the
transpose of the exact forward's matrix, entry by entry, for rays that run up
and down, steep and flat, through volumes of odd and tiny sizes.

The matrix is the exact forward of every unit volume (weights exact up to one
rounding each); a voxel sums at most a few samples of each ray, in any order,
in FP32, so it may be off by 2^-24 for each of its terms -- at most 8 per ray --
and 8 more for a term's products, relative to the sum of the terms' sizes."""
import numpy as np
import pytest
import torch

from curadon_gb300 import ConeGeometry, FanGeometry, adjoint, forward
from curadon_gb300.phantom import cone_config, fan_config

pytestmark = pytest.mark.gpu


def check(geom, shape, dev):
    n = int(np.prod(shape))
    rows = []
    for i in range(n):
        x = torch.zeros(n, device=dev)
        x[i] = 1.0
        ax = torch.zeros(geom.sinogram_shape(), device=dev)
        forward(x.reshape(shape), ax, geom, exact=True)
        rows.append(ax.double().flatten())
    a = torch.stack(rows)  # (voxels, rays)
    y = torch.randn(geom.sinogram_shape(), device=dev, generator=torch.Generator(dev).manual_seed(n))
    y[..., ::5] = 0.0  # rays that are skipped
    out = torch.zeros(shape, device=dev)
    adjoint(y, out, geom)
    want = a @ y.double().flatten()
    size = a.abs() @ y.double().flatten().abs()
    rays = int((a != 0).sum(1).max())
    bound = 2.0 ** -24 * (8 * rays + 8) * size + 1e-30
    assert ((out.double().flatten() - want).abs() <= bound).all()


@pytest.mark.parametrize("algo", ["adj2d=quad", "adj2d=pair"])
@pytest.mark.parametrize("shape,nangles,det", [((1, 1), 5, 4), ((2, 9), 12, 14), ((9, 7), 16, 15),
                                               ((12, 12), 24, 33)])
def test_2d(cuda_device, monkeypatch, algo, shape, nangles, det):
    monkeypatch.setenv("CURADON_GB300_ALGO", algo)
    g = fan_config(max(shape), nangles, det, 1.1)
    g.update(vol_shape=shape)
    check(FanGeometry(**g), shape, cuda_device)


@pytest.mark.parametrize("order", ["view", "band"])
@pytest.mark.parametrize("shape,nangles,det", [((1, 1, 1), 4, 3), ((2, 5, 3), 8, 7),
                                               ((6, 5, 7), 12, 10)])
def test_3d(cuda_device, monkeypatch, order, shape, nangles, det):
    monkeypatch.setenv("CURADON_GB300_ALGO", "adj3d_order=" + order)
    g = cone_config(max(shape), nangles, det)
    g.update(vol_shape=shape)
    check(ConeGeometry(**g), shape, cuda_device)
