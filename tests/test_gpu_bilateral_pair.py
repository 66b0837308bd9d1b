"""The mixed form's filter with two pixels a thread (a table of mixed sessions
alone, large enough) against its one pixel a thread (beside an FP32 session):
the same bits, on ragged images, with holes and without, for the unrolled window
and another."""
import numpy as np
import pytest

from dynamap_b200 import abi, configs
from dynamap_b200.session import Batch, Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(601, 521), (720, 640)])
@pytest.mark.parametrize("diameter,holes", [(8, False), (8, True), (5, True)])
def test_pair_and_single_agree(gpu_lib, rows, cols, diameter, holes):
    p = configs.preset("cfg1")
    p["sensor"].update(rows=rows, cols=cols, fx=525.0, fy=525.0, cx=cols / 2, cy=rows / 2)
    p["tsdf"].update(num_blocks=1 << 14, num_buckets=1 << 15, voxel_size=0.02,
                     truncation_distance=0.08)
    p["bilateral"].update(diameter=diameter)
    rng = np.random.default_rng(rows + diameter)
    d = (1500 + 300 * np.sin(np.arange(cols) / 19.0)[None, :]
         + 200 * np.cos(np.arange(rows) / 13.0)[:, None] + rng.normal(0, 8, (rows, cols)))
    if holes:
        d[rng.random((rows, cols)) < 0.1] = 0
    depth = d.astype(np.uint16)
    t, g, b, s = configs.structs(p)
    alone = Session(t, g, b, s, precision=abi.PRECISION_MIXED_BAND)
    mixed = Session(t, g, b, s, precision=abi.PRECISION_MIXED_BAND)
    plain = Session(t, g, b, s)
    with alone, mixed, plain:
        alone.process(depth)
        batch = Batch([mixed, plain])
        batch.process([depth, depth])
        a = alone.image(1, 0, (rows, cols), np.float32)
        r = mixed.image(1, 0, (rows, cols), np.float32)
        np.testing.assert_array_equal(a.view(np.uint32), r.view(np.uint32))
        assert np.count_nonzero(a) == np.count_nonzero(depth)
        batch.close()


@pytest.mark.parametrize("rows,cols", [(420, 560), (425, 575)])
def test_pair_from_the_smallest_size(gpu_lib, rows, cols):
    """The smallest images with two pixels a thread (tiles of eight rows)."""
    test_pair_and_single_agree(gpu_lib, rows, cols, 8, True)
