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

from conftest import rel_l2
from curadon_gb300 import ConeGeometry, FanGeometry, adjoint, forward
from curadon_gb300.batch import Batch2d
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


def test_adjoint_2d_when_memory_is_short(cuda_device):
    """A plan without room for the quad accumulators (2 x 67 MB) scatters into
    pairs, for good, and leaves no error behind for the next plan."""
    geom, ref = (FanGeometry(**fan_config(2048, 64)) for _ in range(2))
    y = torch.rand(geom.sinogram_shape(), device=cuda_device)
    expect, out = (torch.zeros((2048, 2048), device=cuda_device) for _ in range(2))
    adjoint(y, expect, ref)
    geom.exact_plan
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(max(0, free - (24 << 20)), dtype=torch.uint8, device=cuda_device)
    try:
        adjoint(y, out, geom)
        torch.cuda.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()
    other = FanGeometry(**fan_config(64, 6))  # its creation checks its launch
    small = torch.ones((64, 64), device=cuda_device)
    forward(small, torch.zeros(other.sinogram_shape(), device=cuda_device), other)
    assert rel_l2(out.cpu(), expect.cpu()) < 1e-5
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    adjoint(y, out, geom)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > free - (64 << 20)
    assert rel_l2(out.cpu(), 2 * expect.cpu()) < 1e-5


def test_adjoint_2d_first_used_under_capture(cuda_device):
    geom, ref = (FanGeometry(**fan_config(300, 90)) for _ in range(2))
    y = torch.rand(geom.sinogram_shape(), device=cuda_device)
    expect, out = (torch.zeros((300, 300), device=cuda_device) for _ in range(2))
    adjoint(y, expect, ref)
    geom.exact_plan
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        adjoint(y, out, geom)
    graph.replay()
    adjoint(y, out, geom)  # outside: with its quads
    graph.replay()
    torch.cuda.synchronize()
    assert rel_l2(out.cpu(), 3 * expect.cpu()) < 1e-5


@pytest.mark.parametrize("n,views", [(7, 1), (40, 1), (300, 1), (300, 77), (300, 78), (1300, 1),
                                     (1300, 2), (1800, 8), (1800, 9), (2300, 5), (2300, 6)])
def test_adjoint_2d_of_few_rays(cuda_device, n, views):
    """Few rays scatter sample by sample, more hold their contributions: the
    transpose of the exact forward on both sides of the lines, alone and in a
    batch (on 152 SMs: 912 warps of rays for quads, 608 for pairs)."""
    geom = FanGeometry(**fan_config(n, views))
    gen = torch.Generator(cuda_device).manual_seed(n + views)
    x = torch.rand((n, n), device=cuda_device, generator=gen)
    y = torch.rand(geom.sinogram_shape(), device=cuda_device, generator=gen)
    ax, aty, batched = torch.zeros_like(y), torch.zeros_like(x), torch.zeros_like(x)
    forward(x, ax, geom, exact=True)
    adjoint(y, aty, geom)
    Batch2d([geom], [batched], [y], forward="registers").adjoint()
    torch.cuda.synchronize()
    lhs = float((ax.double() * y.double()).sum())
    for out in (aty, batched):
        assert abs(lhs - float((x.double() * out.double()).sum())) < 1e-5 * abs(lhs)
