"""The texture forward splits a ray's samples into four runs on four lane
groups: against the FP32 register forward, where runs are empty or uneven and
tiles (8 cells x 8 views) have edges."""
import pytest
import torch

from curadon_gb300 import FanGeometry
from curadon_gb300.backend import forward_2d
from curadon_gb300.batch import Batch2d
from curadon_gb300.phantom import fan_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 16, 23])
@pytest.mark.parametrize("views,det", [(1, 1), (7, 9), (8, 8), (9, 7), (33, 40)])
def test_runs(cuda_device, n, views, det):
    geom = FanGeometry(**fan_config(n, views, det))
    vol = torch.rand((n, n), device=cuda_device)
    out = {}
    for algorithm in ("texture", "registers"):
        plan = geom._make_plan()
        plan.set_algorithm(forward=algorithm)
        out[algorithm] = torch.full(geom.sinogram_shape(), -1.0, device=cuda_device)
        forward_2d(vol, out[algorithm], plan)
    batched = torch.full_like(out["texture"], -2.0)
    Batch2d([geom], [vol], [batched], forward="texture").forward()
    torch.cuda.synchronize()
    assert torch.equal(batched, out["texture"])
    # the texture unit rounds its two weights to 8 bits: at most 2^-9 of the
    # texels' range (1) per weight and sample, n + 1 samples of length up to
    # sqrt(2); a lost or doubled sample is 0.5 on average
    assert float((out["texture"] - out["registers"]).abs().max()) <= 2 * 2.0 ** -9 * (n + 1) * 1.4143
