"""The 2D register forward in bundles takes every ray's samples in the ray's own
order and in the ray-by-ray kernel's operations: equal bits, alone and in a
batch, where bundles have edges (64 cells, 4 views), rays of one bundle go both
ways or the source lies close to (or inside) the image."""
import numpy as np
import pytest
import torch

from curadon_gb300 import FanGeometry, FanVecGeometry, forward
from curadon_gb300.backend import forward_2d
from curadon_gb300.batch import Batch2d
from curadon_gb300.phantom import fan_config

pytestmark = pytest.mark.gpu


def geometries():
    for n, views, det in ((33, 7, 50), (64, 3, 63), (64, 4, 64), (100, 5, 65), (257, 37, 364),
                          (1024, 21, 1449)):
        yield f"{n}", FanGeometry(**fan_config(n, views, det))
    for dso, dsd, ds in ((80, 100, 2.0), (66, 400, 30.0), (30, 60, 3.0)):  # wide; inside
        yield f"wide {dso}", FanGeometry(**fan_config(100, 90, 211, ds, dso, dsd))
    g = dict(fan_config(48, 37, 70, 1.3, 90.0, 150.0), vol_shape=(48, 60), vol_spacing=(0.9, 1.2),
             vol_offset=(2.0, -3.0), det_offset=1.5)
    yield "offsets", FanGeometry(**g)
    g = fan_config(300, 77)
    v = np.asarray(FanGeometry(**g).to_vec())
    v[:, 4:] *= g["det_spacing"]
    v[::2] = np.concatenate([v[::2, :4] * [-1, -1, -1, -1], v[::2, 4:]], axis=1)  # both ways
    yield "vectors", FanVecGeometry((300, 200), g["det_shape"], v)


@pytest.mark.parametrize("name,geom", [pytest.param(n, g, id=n) for n, g in geometries()])
def test_bundled_register_forward(cuda_device, monkeypatch, name, geom):
    gen = torch.Generator(device=cuda_device).manual_seed(len(name))
    vol = torch.rand(tuple(int(v) for v in geom.vol_shape), device=cuda_device, generator=gen)
    alone = torch.full(geom.sinogram_shape(), -1.0, device=cuda_device)
    batched, rays = torch.full_like(alone, -2.0), torch.full_like(alone, -3.0)
    forward(vol, alone, geom, exact=True)
    Batch2d([geom], [vol], [batched], forward="registers").forward()
    monkeypatch.setenv("CURADON_GB300_ALGO", "fwd2d=alu,fwd2d_march=off")
    plan = geom._make_plan()
    monkeypatch.delenv("CURADON_GB300_ALGO")
    forward_2d(vol, rays, plan)
    torch.cuda.synchronize()
    assert torch.equal(alone, rays)
    assert torch.equal(batched, rays)


@pytest.mark.parametrize("n", [6000, 8192, 16384])
def test_bundled_register_forward_of_wide_images(cuda_device, monkeypatch, n):
    """A ray's column is a running sum, which at these sizes strays from its line
    by a column and more: the bundle's windows hold those samples too."""
    g = fan_config(n, 8, 3 * n // 2)
    g["angles"] = (0.0007 * np.arange(8)).astype(np.float32)  # windows within their buffers
    geom = FanGeometry(**g)
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    vol = torch.rand((n, n), device=cuda_device, generator=gen)
    alone = torch.full(geom.sinogram_shape(), -1.0, device=cuda_device)
    rays = torch.full_like(alone, -3.0)
    forward(vol, alone, geom, exact=True)
    monkeypatch.setenv("CURADON_GB300_ALGO", "fwd2d=alu,fwd2d_march=off")
    plan = geom._make_plan()
    monkeypatch.delenv("CURADON_GB300_ALGO")
    forward_2d(vol, rays, plan)
    torch.cuda.synchronize()
    assert torch.equal(alone, rays)


def test_forward_block_shapes_the_ray_by_ray_kernel(cuda_device, monkeypatch):
    g = FanGeometry(**fan_config(100, 37, 211))
    vol = torch.rand((100, 100), device=cuda_device)
    expect = forward(vol, torch.zeros(g.sinogram_shape(), device=cuda_device), g, exact=True)
    monkeypatch.setenv("CURADON_GB300_ALGO", "fwd2d=alu,fwd2d_march=off")
    plan = g._make_plan()
    for bx, by in ((32, 8), (64, 2), (256, 1), (32, 1)):
        plan.forward_block_y = 1
        plan.forward_block_x, plan.forward_block_y = bx, by
        assert (plan.forward_block_x, plan.forward_block_y) == (bx, by)
        out = torch.full_like(expect, -1.0)
        forward_2d(vol, out, plan)
        assert torch.equal(out, expect)


@pytest.mark.parametrize("count", [2, 40])  # in bundles; too many of them: ray by ray
def test_small_problems_of_a_batch(cuda_device, count):
    geoms = [FanGeometry(**fan_config(72 + k % 3, 120)) for k in range(count)]
    gen = torch.Generator(device=cuda_device).manual_seed(count)
    vols = [torch.rand(tuple(int(v) for v in g.vol_shape), device=cuda_device, generator=gen)
            for g in geoms]
    sinos = [torch.full(g.sinogram_shape(), -1.0, device=cuda_device) for g in geoms]
    Batch2d(geoms, vols, sinos, forward="registers").forward()
    for g, v, s in zip(geoms, vols, sinos):
        assert torch.equal(s, forward(v, torch.full_like(s, -2.0), g, exact=True))
