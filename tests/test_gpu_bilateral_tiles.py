"""dyn_bilateral_filter at the edges of its tiles and branches: images smaller
than a tile, one off a tile's size, both tile heights; every window parity of
the unrolled rows; depths that span little (the exponent's reduction left
out) and widely (small range sigma: kept); images with holes, without, and
with NaN, infinite and negative depths.  Bit for bit the oracle's, which runs
the same operations in the same order."""
import ctypes as C

import numpy as np
import pytest

from dynamap_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (4, 32), (5, 33), (17, 95), (121, 163), (240, 967)])
@pytest.mark.parametrize("diameter,sigma_i", [(8, 10.0), (8, 0.05), (1, 10.0), (5, 10.0), (16, 0.3)])
def test_filter_bits(gpu_lib, oracle, rows, cols, diameter, sigma_i):
    import torch
    rng = np.random.default_rng(rows * 1000 + cols)
    base = (1.5 + 0.4 * np.sin(np.arange(cols) / 9.0)[None, :] + 0.2 * np.cos(np.arange(rows) / 7.0)[:, None]
            + rng.normal(0, 0.01, (rows, cols))).astype(np.float32)
    holes = np.where(rng.random((rows, cols)) < 0.1, np.float32(0), base).astype(np.float32)
    odd = holes.copy()
    odd.ravel()[:: 97] = np.float32(-1.0)
    odd.ravel()[1:: 211] = np.float32("nan")
    p = abi.BilateralParams(diameter, sigma_i, 1.0, 1)
    for d in (base, holes, odd):
        src = torch.from_numpy(d).cuda()
        out = torch.empty_like(src)
        abi.check("dyn_bilateral_filter", gpu_lib.dyn_bilateral_filter(
            src.data_ptr(), out.data_ptr(), rows, cols, C.byref(p), None))
        torch.cuda.synchronize()
        ref = oracle.bilateral(d, p)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("rows,cols", [(17, 95), (121, 163)])
@pytest.mark.parametrize("diameter,sigma_i", [(8, 10.0), (8, 0.05), (5, 10.0)])
def test_filter_with_infinite_depths(gpu_lib, oracle, rows, cols, diameter, sigma_i):
    """Infinite depths: isolated ones, and a stretch of tiles with no other valid
    pixel, whose span of depths is inf - inf.  The oracle's bits; where its value
    is NaN (an infinite depth's weight is zero), a NaN."""
    import torch
    rng = np.random.default_rng(rows + diameter)
    d = rng.uniform(1.0, 2.0, (rows, cols)).astype(np.float32)
    d.ravel()[5::113] = np.inf
    d[rows // 2:, cols // 2:] = 0
    d[rows // 2 + 2::5, cols // 2 + 3::7] = np.inf
    p = abi.BilateralParams(diameter, sigma_i, 1.0, 1)
    src = torch.from_numpy(d).cuda()
    out = torch.empty_like(src)
    abi.check("dyn_bilateral_filter", gpu_lib.dyn_bilateral_filter(
        src.data_ptr(), out.data_ptr(), rows, cols, C.byref(p), None))
    torch.cuda.synchronize()
    got, ref = out.cpu().numpy(), oracle.bilateral(d, p)
    nan = np.isnan(ref)
    assert nan.any() and np.isfinite(ref[ref != 0]).any()
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint32), ref[~nan].view(np.uint32))
