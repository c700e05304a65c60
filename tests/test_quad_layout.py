"""GPU test of the quad copies written in 32-column, 8-row pieces: the axial
backprojection, which reads them, equals the general kernel, which reads
8-byte pairs laid out one by one, at detectors around the pieces' edges.

Both take the same bilinear samples; a coordinate (up to cells + voxels) may
differ by 8 roundings of 2^-23 of its size, a sample then by twice that (two
axes, slopes up to the largest value 1), and by as much for its own sums."""
import pytest
import torch

from curadon_gb300 import ConeGeometry, backward
from curadon_gb300.phantom import cone_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,views", [(5, 3), (18, 9)])
@pytest.mark.parametrize("det", [(1, 1), (4, 28), (5, 29), (12, 27), (28, 60), (13, 61)])
def test_axial_equals_general(cuda_device, monkeypatch, n, views, det):
    g = cone_config(n, views, 1)
    g.update(det_shape=det)
    y = torch.rand((views, *det), device=cuda_device,
                   generator=torch.Generator(cuda_device).manual_seed(det[1]))
    out = []
    for algo in ("ax8m5", "pair"):
        monkeypatch.setenv("CURADON_GB300_ALGO", "bwd3d=" + algo)
        v = torch.zeros((n, n, n), device=cuda_device)
        backward(y, v, ConeGeometry(**g))
        out.append(v.double())
    assert out[1].abs().max() > 0
    assert (out[0] - out[1]).abs().max() <= views * 2.0 ** -18 * (max(det) + n)


@pytest.mark.parametrize("views", [63, 64])  # a warp's 8 x 4 and 4 x 8 voxels
@pytest.mark.parametrize("shape", [(1, 1, 1), (9, 3, 31), (7, 9, 33), (17, 8, 70)])
def test_axial_patches_cover_the_volume(cuda_device, monkeypatch, shape, views):
    n, det = max(shape), (19, 45)
    g = cone_config(n, views, 1)
    g.update(vol_shape=shape, det_shape=det)
    y = torch.rand((views, *det), device=cuda_device,
                   generator=torch.Generator(cuda_device).manual_seed(n))
    out = []
    for algo in ("ax8m5", "pair"):
        monkeypatch.setenv("CURADON_GB300_ALGO", "bwd3d=" + algo)
        v = torch.zeros(shape, device=cuda_device)
        backward(y, v, ConeGeometry(**g))
        out.append(v.double())
    assert out[1].abs().max() > 0
    assert (out[0] - out[1]).abs().max() <= views * 2.0 ** -18 * (max(det) + n)
