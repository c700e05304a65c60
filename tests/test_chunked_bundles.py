"""The chunked 2D forward's two bundle sizes take the same samples in the same
order, so their results are equal bit for bit -- at the edges of the bundles
(64 / 128 cells, 4 / 8 views), where windows outgrow their buffers (few views
over a full turn) and in batches."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from curadon_gb300 import FanGeometry, forward
from curadon_gb300.batch import Batch2d
from curadon_gb300.phantom import ellipses_2d, fan_config

pytestmark = pytest.mark.gpu

CASES = [(705, 3, 63), (720, 4, 64), (704, 5, 65), (710, 9, 129), (1024, 37, 1449), (800, 200, 1131)]


def geometry(monkeypatch, bundle, n, views, det):
    monkeypatch.setenv("CURADON_GB300_ALGO", f"fwd2d_bundle={bundle}")
    geom = FanGeometry(**fan_config(n, views, det))
    assert geom.plan.algorithm[0] == "chunked"
    monkeypatch.delenv("CURADON_GB300_ALGO")
    return geom


@pytest.mark.parametrize("n,views,det", CASES)
def test_bundles_agree(cuda_device, monkeypatch, n, views, det):
    vol = ellipses_2d(n, n + views, device=cuda_device).contiguous()
    out = {}
    for bundle in ("small", "large"):
        geom = geometry(monkeypatch, bundle, n, views, det)
        out[bundle] = torch.full(geom.sinogram_shape(), -1.0, device=cuda_device)
        forward(vol, out[bundle], geom)
    torch.cuda.synchronize()
    assert torch.equal(out["small"], out["large"])
    import oracle

    # 1e-3: the operators' parity bar
    assert rel_l2(out["small"].cpu(), oracle.fwd2d(fan_config(n, views, det), vol.cpu().numpy())) < 1e-3


def test_batched_bundles_agree(cuda_device, monkeypatch):
    geoms, vols, sinos, expect = [], [], [], []
    for k, (n, views, det) in enumerate(CASES):
        bundle = ("small", "large")[k % 2]
        vols.append(ellipses_2d(n, k, device=cuda_device).contiguous())
        geoms.append(geometry(monkeypatch, bundle, n, views, det))
        sinos.append(torch.zeros(geoms[-1].sinogram_shape(), device=cuda_device))
        expect.append(forward(vols[-1], torch.zeros_like(sinos[-1]), geoms[-1]))
    Batch2d(geoms, vols, sinos, forward="plans").forward()
    torch.cuda.synchronize()
    for s, e in zip(sinos, expect):
        assert torch.equal(s, e)


@pytest.mark.parametrize("n,angle", [(6000, 2.0), (8192, 2.0), (16384, 0.4)])
def test_bundles_of_wide_images_agree(cuda_device, monkeypatch, n, angle):
    """Both bundles' windows hold the samples whose columns, running sums, have
    strayed from their rays' lines, and those that strayed off the padding."""
    g = fan_config(n, 8, 3 * n // 2)
    g["angles"] = (angle + 0.0007 * np.arange(8)).astype(np.float32)
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    vol = torch.rand((n, n), device=cuda_device, generator=gen)
    out = []
    for bundle in ("small", "large"):
        monkeypatch.setenv("CURADON_GB300_ALGO", f"fwd2d_bundle={bundle}")
        geom = FanGeometry(**g)
        assert geom.plan.algorithm[0] == "chunked"
        monkeypatch.delenv("CURADON_GB300_ALGO")
        out.append(forward(vol, torch.full(geom.sinogram_shape(), -1.0, device=cuda_device), geom))
    torch.cuda.synchronize()
    assert torch.equal(*out)
