"""The 2D backprojection's split of the views: the direct kernel (small
images), the clusters (views in groups on several thread blocks) and the
batched tiles (groups in turn) sum each pixel's views in the same groups and
order, so a batch of one problem equals the single call bit for bit."""
import pytest
import torch

from conftest import rel_l2
from curadon_gb300 import FanGeometry, backward
from curadon_gb300.batch import Batch2d
from curadon_gb300.phantom import fan_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,views,det", [
    ((1, 1), 1, 1), ((8, 8), 32, 12), ((9, 17), 33, 26), ((64, 64), 360, 91),       # direct
    ((33, 70), 1100, 100), ((158, 159), 512, 226), ((161, 160), 512, 227),          # its limit
    ((512, 65), 600, 725), ((257, 255), 290, 364), ((640, 640), 223, 906),          # clusters
    ((700, 1100), 64, 1301), ((900, 900), 450, 1273)])                              # one group
def test_split_views_equal_groups_in_turn(cuda_device, shape, views, det):
    n = max(shape)
    g = dict(fan_config(n, views, det, DSO=2.0 * n + 4, DSD=3.0 * n + 8), vol_shape=shape)
    geom = FanGeometry(**g)
    gen = torch.Generator(device=cuda_device).manual_seed(n + views)
    y = torch.rand(geom.sinogram_shape(), device=cuda_device, generator=gen)
    start = torch.rand(shape, device=cuda_device, generator=gen)
    alone, batched = start.clone(), start.clone()
    backward(y, alone, geom)
    Batch2d([geom], [batched], [y]).backward()
    torch.cuda.synchronize()
    assert torch.equal(alone, batched)
    import oracle

    # 1e-3: the operators' parity bar
    ref = oracle.bwd2d(g, y.cpu().numpy(), vol0=start.cpu().numpy())
    assert rel_l2(alone.cpu(), ref) < 1e-3


@pytest.mark.parametrize("n,views", [(64, 360), (300, 400)])
def test_split_views_nonfinite(cuda_device, n, views):
    """An infinite or NaN cell reaches the same pixels either way."""
    geom = FanGeometry(**fan_config(n, views))
    y = torch.rand(geom.sinogram_shape(), device=cuda_device)
    y[views // 3, 40], y[views // 2, 50] = float("inf"), float("nan")
    alone, batched = (torch.zeros((n, n), device=cuda_device) for _ in range(2))
    backward(y, alone, geom)
    Batch2d([geom], [batched], [y]).backward()
    torch.cuda.synchronize()
    assert torch.equal(torch.isnan(alone), torch.isnan(batched))
    assert torch.equal(torch.nan_to_num(alone), torch.nan_to_num(batched))


@pytest.mark.parametrize("n,views", [(64, 360), (120, 700), (300, 400), (640, 640), (900, 450),
                                     (800, 33), (600, 48)])
def test_a_large_volume_is_rounded_once(cuda_device, n, views):
    """However many groups a pixel's views are summed in, a value that the volume
    holds already takes one rounding of the result (2^-24 of it) and one of the
    backprojection itself."""
    geom = FanGeometry(**fan_config(n, views))
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    y = torch.rand(geom.sinogram_shape(), device=cuda_device, generator=gen)
    start = 1e6 + torch.rand((n, n), device=cuda_device, generator=gen)
    plain = torch.zeros_like(start)
    backward(y, plain, geom)
    alone, batched = start.clone(), start.clone()
    backward(y, alone, geom)
    Batch2d([geom], [batched], [y]).backward()
    torch.cuda.synchronize()
    exact = start.double() + plain.double()
    bound = 2.0 ** -24 * (1.0001 * exact.abs() + plain.double().abs())
    for out in (alone, batched):
        assert bool(((out.double() - exact).abs() <= bound).all())
