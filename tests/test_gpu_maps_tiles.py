"""Vertices and normals of one level (dyn_depth_to_maps) in each tile shape:
images as wide as a tile or a pixel beside it, narrow and wide strips, a
vertex map or none.  Bit for bit the oracle's."""
import ctypes as C

import numpy as np
import pytest

from dynamap_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(64, 128), (63, 129), (40, 103), (7, 102), (33, 32), (50, 33),
                                       (65, 40), (31, 26), (70, 25), (130, 8), (129, 9), (300, 5),
                                       (3, 700), (2, 5), (1, 1)])
def test_maps_in_each_tile_shape(gpu_lib, oracle, rows, cols):
    import torch
    rng = np.random.default_rng(rows * 1000 + cols)
    d = rng.uniform(0.5, 4.0, (rows, cols)).astype(np.float32)
    d[rng.random((rows, cols)) < 0.1] = 0
    f = max(60.0, 525.0 * cols / 640.0)
    s = abi.Sensor(rows=rows, cols=cols, fx=f, fy=f, cx=(cols - 1) / 2, cy=(rows - 1) / 2,
                   depth_scaler=1000.0)
    ov, on = oracle.maps(d, s)
    dd = torch.from_numpy(d).cuda()
    for vertices in (True, False):
        v = torch.full((rows, cols, 4), 7.0, device="cuda")
        n = torch.full((rows, cols, 4), 7.0, device="cuda")
        abi.check("dyn_depth_to_maps", gpu_lib.dyn_depth_to_maps(
            dd.data_ptr(), C.byref(s), v.data_ptr() if vertices else None, n.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        np.testing.assert_array_equal(n.cpu().numpy().view(np.uint32),
                                      np.asarray(on).view(np.uint32))
        if vertices:
            np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32),
                                          np.asarray(ov).view(np.uint32))
        else:
            assert (v == 7.0).all()
