"""GPU test of half inputs read where they are laid out: every 2D algorithm on
half volumes and sinograms gives its own FP32 result on the same values,
rounded once, at odd sizes and from addresses aligned to 2 bytes only."""
import pytest
import torch

from curadon_gb300 import FanGeometry
from curadon_gb300.backend import backward_2d, forward_2d
from curadon_gb300.phantom import fan_config

pytestmark = pytest.mark.gpu


def halves(shape, dev, seed):
    """Half values that start 2 bytes past an aligned address."""
    n = shape[0] * shape[1]
    g = torch.Generator(dev).manual_seed(seed)
    return torch.rand(n + 1, device=dev, generator=g).half()[1:].view(shape)


@pytest.mark.parametrize("shape,views,det", [((1, 1), 1, 1), ((33, 47), 9, 61), ((64, 64), 40, 91),
                                             ((300, 211), 130, 333)])
@pytest.mark.parametrize("algorithm", [("registers", "registers"), ("texture", "texture"),
                                       ("chunked", "shared")])
def test_rounded_fp32(cuda_device, shape, views, det, algorithm):
    g = fan_config(max(shape), views, det)
    g.update(vol_shape=shape)
    plans = {}
    for bits in (16, 32):
        plans[bits] = FanGeometry(**g, vol_prec=bits, sino_prec=bits)._make_plan()
        plans[bits].set_algorithm(forward=algorithm[0], backward=algorithm[1])
    x, y = halves(shape, cuda_device, 1), halves((views, det), cuda_device, 2)
    out = {}
    for bits, dtype in ((16, torch.float16), (32, torch.float32)):
        s = torch.zeros((views, det), device=cuda_device, dtype=dtype)
        v = torch.zeros(shape, device=cuda_device, dtype=dtype)
        forward_2d(x.to(dtype) if bits == 32 else x, s, plans[bits])
        backward_2d(v, y.to(dtype) if bits == 32 else y, plans[bits])
        out[bits] = (s, v)
    # one half of the pair only
    mixed = torch.zeros((views, det), device=cuda_device)
    forward_2d(x, mixed, plans[16])
    back = torch.zeros(shape, device=cuda_device)
    backward_2d(back, y, plans[32])
    torch.cuda.synchronize()
    assert torch.equal(out[16][0], out[32][0].half())
    assert torch.equal(out[16][1], out[32][1].half())
    assert torch.equal(mixed, out[32][0])
    assert torch.equal(back, out[32][1])
