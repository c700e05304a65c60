"""The 64-bit rays of the performance cases are finite, also those that miss the
image or only touch its corner: their positions become indices."""
import importlib.util
import random
from pathlib import Path

import pytest
import torch

spec = importlib.util.spec_from_file_location(
    "perf_cases", Path(__file__).resolve().parent.parent / "perf" / "cases.py")
cases = importlib.util.module_from_spec(spec)
spec.loader.exec_module(cases)


def drawn():
    yield cases.fan("", "forward", 78, 78, 111)  # one ray through a corner alone
    for seed in range(40):
        c = cases.draw(random.Random(seed))
        if not c["op"].startswith("cone_") and c["op"] != "batch" and c["det"] * c["views"] < 2e5:
            yield c


@pytest.mark.parametrize("case", [pytest.param(c, id=f"{c['height']}x{c['width']}-{c['det']}")
                                  for c in drawn()])
def test_fan_rays_are_finite(case):
    rays = cases.FanRays(case, cases.fan_vectors(case, 1), torch.device("cpu"))
    for t in (*rays.p, *rays.v, rays.steps, rays.norm):
        assert bool(torch.isfinite(t).all())


def test_a_touching_ray_adds_nothing():
    case = cases.fan("", "forward", 78, 78, 111)
    v = cases.fan_vectors(case, 1)
    y = cases.fan_forward64(case, v, torch.ones((78, 78)))
    assert bool(torch.isfinite(y).all()) and float(y.max()) > 78
    assert bool(torch.isfinite(cases.fan_adjoint64(case, v, y)).all())
