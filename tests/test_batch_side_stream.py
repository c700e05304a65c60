"""GPU test of the batched "plans" forward, whose chunked problems run on a
side stream beside the texture ones: the bits of the single problems, on the
default and on another stream, followed at once by work that reads the
sinograms and rewrites the volumes, and replayed from a graph."""
import pytest
import torch

from curadon_gb300 import FanGeometry
from curadon_gb300.backend import forward_2d
from curadon_gb300.batch import Batch2d
from curadon_gb300.phantom import fan_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [["chunked"], ["texture"], ["chunked", "texture"],
                                   ["texture", "chunked", "texture", "chunked"]])
@pytest.mark.parametrize("mode", ["default", "stream", "graph"])
def test_bits(cuda_device, kinds, mode):
    geoms, vols, sinos, want = [], [], [], []
    for k, kind in enumerate(kinds):
        n = (40, 131, 256, 97)[k]
        geom = FanGeometry(**fan_config(n, 30 + 7 * k))
        geom.plan.set_algorithm(forward=kind)
        geoms.append(geom)
        vols.append(torch.rand((n, n), device=cuda_device))
        sinos.append(torch.zeros(geom.sinogram_shape(), device=cuda_device))
        want.append(torch.zeros_like(sinos[-1]))
        forward_2d(vols[-1], want[-1], geom.plan)
    batch = Batch2d(geoms, vols, sinos, forward="plans")
    keep = [v.clone() for v in vols]
    copies = [torch.empty_like(s) for s in sinos]

    def step():  # twice: the second call writes the same scratch as the first
        for _ in range(2):
            for v, k in zip(vols, keep):
                v.copy_(k)
            batch.forward()
            for c, s in zip(copies, sinos):
                c.copy_(s)
            for v in vols:
                v.zero_()
        batch.backward()  # dependent launches right behind the join

    torch.cuda.synchronize()
    if mode == "default":
        step()
    else:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            step()
        side.synchronize()
        if mode == "graph":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step()
            for c in copies:
                c.zero_()
            for _ in range(2):
                graph.replay()
    torch.cuda.synchronize()
    for c, w in zip(copies, want):
        assert torch.equal(c, w)
