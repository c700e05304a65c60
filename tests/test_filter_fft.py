"""The row filter by FFT (long rows, ramp-like taps) against 64 bits: at the
edges of its transform sizes, beside rows it leaves to the direct sum."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from curadon_gb300.fbp import filter_kernel, filter_sinogram

pytestmark = pytest.mark.gpu

# two transforms of at most 12 rounding levels (rms 1e-7 each of their input)
# and |d| max|G| / |result| about 2 (the spectrum of a ramp's running sums lies
# between 1/pi and 1/2): 4e-7, with a margin of 5
TOL = 2e-6


def exact(rows, name, scale=1.0, pre=None):
    h = filter_kernel(rows.shape[-1], name).astype(np.float32).astype(np.float64)
    x = rows.double().cpu().numpy() * (1.0 if pre is None else pre.double().cpu().numpy())
    return scale * np.fft.irfft(np.fft.rfft(x) * np.fft.rfft(h), n=rows.shape[-1])


def rel(a, b):
    return np.linalg.norm(a.double().cpu().numpy() - b) / np.linalg.norm(b)


@pytest.mark.parametrize("cells", [159, 160, 161, 511, 512, 513, 1024, 1025, 1449, 2048, 2049,
                                   4095, 4096, 4097])
@pytest.mark.parametrize("rows", [47, 48, 131])
def test_filter_sizes(cuda_device, cells, rows):
    gen = torch.Generator(device=cuda_device).manual_seed(cells + rows)
    s = torch.rand((rows, cells), device=cuda_device, generator=gen)
    # (the direct sum's running error over thousands of terms: 1e-5)
    tol = TOL if rows >= 48 and 160 <= cells <= 4096 else 1e-5
    assert rel(filter_sinogram(s, "ram-lak", scale=0.3), exact(s, "ram-lak", 0.3)) < tol


@pytest.mark.parametrize("name", ["shepp-logan", "hamming", "hann"])
def test_filter_windows_and_weights(cuda_device, name):
    s = torch.rand((3, 50, 363), device=cuda_device)
    pre = 0.5 + torch.rand(363, device=cuda_device)
    out = filter_sinogram(s, name, scale=2.0, pre_weight=pre)
    assert rel(out, exact(s, name, 2.0, pre)) < TOL


def test_taps_with_a_response_at_zero_stay_direct(cuda_device):
    s = torch.rand((64, 725), device=cuda_device)
    out = filter_sinogram(s, None, scale=0.5)  # an impulse, and 64-bit rounding noise of 1e-17
    assert torch.equal(out, 0.5 * s)


def test_rows_do_not_meet(cuda_device):
    """Rows of any size, infinite or NaN leave the others as they are."""
    s = torch.rand((60, 725), device=cuda_device)
    clean = filter_sinogram(s, "ram-lak")
    odd = s.clone()
    odd[3, 100], odd[7, 5], odd[20] = float("inf"), float("nan"), odd[20] * 1e33
    odd[40] = 0.0
    out = filter_sinogram(odd, "ram-lak")
    keep = [i for i in range(60) if i not in (3, 7, 20, 40)]
    assert torch.equal(out[keep], clean[keep])
    assert bool((out[40] == 0).all()) and bool(torch.isnan(out[7]).all())
    assert not bool(torch.isfinite(out[3]).any())
    assert rel(out[20:21] * 1e-33, exact(odd[20:21] * 1e-33, "ram-lak")) < 1e-5


@pytest.mark.parametrize("cells", [160, 363, 725, 1449, 4096])
def test_a_row_is_filtered_alike_in_any_stack(cuda_device, cells):
    s = torch.rand((131, cells), device=cuda_device)
    stack = filter_sinogram(s, "ram-lak")
    for rows in (1, 5, 47, 48):
        assert torch.equal(filter_sinogram(s[:rows].clone(), "ram-lak"), stack[:rows])
        assert torch.equal(filter_sinogram(s[-rows:].clone(), "ram-lak"), stack[-rows:])


@pytest.mark.parametrize("rows,cells", [(1031, 1449), (2051, 2897), (5003, 363), (1301, 4096)])
def test_blocks_that_walk_over_rows(cuda_device, rows, cells):
    """More rows than the resident blocks take at once, with a remainder."""
    s = torch.rand((rows, cells), device=cuda_device)
    out = filter_sinogram(s, "ram-lak")
    assert rel(out, exact(s, "ram-lak")) < TOL
    for part in (out[:7], out[rows // 2:rows // 2 + 7], out[-7:]):  # and each part by itself
        i = (part.data_ptr() - out.data_ptr()) // (4 * cells)
        assert rel(part, exact(s[i:i + 7], "ram-lak")) < TOL


@pytest.mark.parametrize("rows,cells", [(2003, 725), (5003, 363), (2001, 1449)])
def test_rows_do_not_meet_over_rounds(cuda_device, rows, cells):
    """A block sums some rows directly (infinite, NaN, very large) between others."""
    s = torch.rand((rows, cells), device=cuda_device)
    clean = filter_sinogram(s, "ram-lak")
    odd = s.clone()
    at = [0, 3, 17, rows // 2, rows // 2 + 1, rows - 2]
    odd[at[0], 5], odd[at[1], 100], odd[at[2]] = float("nan"), float("inf"), odd[at[2]] * 1e33
    odd[at[3], 7], odd[at[4]], odd[at[5]] = -float("inf"), odd[at[4]] * 1e33, 0.0
    out = filter_sinogram(odd, "ram-lak")
    keep = [i for i in range(rows) if i not in at]
    assert torch.equal(out[keep], clean[keep])
    for i in (at[2], at[4]):
        assert rel(out[i:i + 1] * 1e-33, exact(odd[i:i + 1] * 1e-33, "ram-lak")) < 1e-5
    assert not bool(torch.isfinite(out[[at[0], at[1], at[3]]]).any())
    assert bool((out[at[5]] == 0).all())


def test_packed_direct_sum_equals_scalar(cuda_device, tmp_path):
    """The direct sum's two kernels (rows too short for the transform; taps with a
    response at zero frequency) agree bit for bit."""
    code = """
import ctypes as C, sys
import numpy as np, torch
from curadon_gb300._lib import check, load
from curadon_gb300.fbp import filter_sinogram
gen = torch.Generator(device="cuda").manual_seed(1)
out = []
for rows, cells in ((37, 150), (37, 1449), (64, 363)):
    s = torch.rand((rows, cells), device="cuda", generator=gen)
    h = torch.rand(cells, device="cuda", generator=gen)
    o = torch.empty_like(s)
    check(load().cg_filter_rows(s.data_ptr(), o.data_ptr(), h.data_ptr(), None, rows, cells, 0.5,
                                torch.cuda.current_stream().cuda_stream))
    out += [o.flatten(), filter_sinogram(s[:, :150].contiguous(), "shepp-logan").flatten()]
np.save(sys.argv[1], torch.cat(out).cpu().numpy())
"""
    got = []
    for mode in ("packed", "scalar"):
        path = tmp_path / f"{mode}.npy"
        subprocess.run([sys.executable, "-c", code, str(path)], check=True, timeout=300,
                       env=dict(os.environ, CURADON_GB300_FILTER=mode))
        got.append(np.load(path))
    assert np.array_equal(*got)
