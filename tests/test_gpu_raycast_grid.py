"""The raycast through the block grid and through the hash give the same bits:
a session whose rays reach a box too large for a grid (long sensor range)
against one with a grid, on ragged images and poses of either sign, in the
three voxel forms; the FP32 form also against the oracle."""
import numpy as np
import pytest

from dynamap_b200 import abi, configs
from dynamap_b200.session import Session

pytestmark = pytest.mark.gpu


def session(p, dmax, prec, frames):
    p["tsdf"].update(max_sensor_depth=dmax)
    t, g, b, s = configs.structs(p)
    m = Session(t, g, b, s, precision=prec)
    for d, c, q in frames:
        m.integrate_with_pose(d, c, q)
    return m, t, s


@pytest.mark.parametrize("prec", [abi.PRECISION_FP32, abi.PRECISION_MIXED,
                                  abi.PRECISION_MIXED_BAND])
@pytest.mark.parametrize("rows,cols,shift", [(61, 83, 0.0), (120, 160, -6.0), (33, 47, -3.0)])
def test_grid_and_hash_marches_agree(gpu_lib, oracle, prec, rows, cols, shift):
    p = configs.preset("cfg2")
    fx = 525.0 * cols / 640.0
    p["sensor"].update(rows=rows, cols=cols, fx=fx, fy=fx, cx=(cols - 1) / 2, cy=(rows - 1) / 2)
    p["tsdf"].update(num_blocks=1 << 14, num_buckets=1 << 15, voxel_size=0.01,
                     truncation_distance=0.04)
    p["gn"].update(lvl_scale=[1, 1, 1])
    seq = configs.sequence(p, seed=17, n_frames=3)
    poses = seq.poses.astype(np.float32)
    poses[:, :3, 3] += np.float32(shift)  # across and beyond the origin
    frames = [(seq.depth[k], seq.rgb[k], poses[k]) for k in range(3)]
    # both ranges take every depth of the frames (up to 4 m): the same maps
    near, t, s = session(p, 6.0, prec, frames)
    far, _, _ = session(p, 60.0, prec, frames)
    with near, far:
        for q in (poses[2], poses[0], np.eye(4, dtype=np.float32)):
            gd, gc = near.raycast(q, rgb=True)
            hd, hc = far.raycast(q, rgb=True)
            hit = gd < 6.0
            np.testing.assert_array_equal(hit, hd < 6.0)
            np.testing.assert_array_equal(gd[hit].view(np.uint32), hd[hit].view(np.uint32))
            np.testing.assert_array_equal(gc[hit], hc[hit])
        assert np.count_nonzero(near.raycast(poses[2])[0] < 6.0) > 0.2 * rows * cols
        if prec == abi.PRECISION_FP32:
            ovol = oracle.Volume(t)
            for d, c, q in frames:
                m = oracle.depth_from_raw(d, s.depth_scaler)
                ovol.allocate(m, s, q)
                ovol.integrate(m, c, s, q)
            for q in (poses[2], poses[0]):
                gd, gc = near.raycast(q, rgb=True)
                od, oc, _ = ovol.raycast(q, s, rgb=True)
                np.testing.assert_array_equal(gd.view(np.uint32), od.view(np.uint32))
                np.testing.assert_array_equal(gc, oc)


@pytest.mark.parametrize("prec", [abi.PRECISION_FP32, abi.PRECISION_MIXED,
                                  abi.PRECISION_MIXED_BAND])
def test_small_views_agree(gpu_lib, prec):
    """Views on either side of the size from which the mixed forms take the grid."""
    p = configs.preset("cfg1")
    p["sensor"].update(rows=120, cols=160, fx=131.25, fy=131.25, cx=79.5, cy=59.5)
    p["tsdf"].update(num_blocks=1 << 14, num_buckets=1 << 15, voxel_size=0.01,
                     truncation_distance=0.04)
    p["gn"].update(lvl_scale=[1, 1, 1])
    seq = configs.sequence(p, seed=23, n_frames=2)
    frames = [(seq.depth[k], None, seq.poses[k].astype(np.float32)) for k in range(2)]
    near, _, _ = session(p, 6.0, prec, frames)
    far, _, _ = session(p, 60.0, prec, frames)
    with near, far:
        for rows, cols in ((15, 17), (16, 16), (6, 8), (1, 1), (24, 32)):
            f = 131.25 * cols / 160.0
            v = abi.Sensor(rows=rows, cols=cols, fx=f, fy=f, cx=(cols - 1) / 2, cy=(rows - 1) / 2,
                           depth_scaler=1000.0)
            a, b = near.raycast(frames[1][2], v)[0], far.raycast(frames[1][2], v)[0]
            hit = a < 6.0
            np.testing.assert_array_equal(hit, b < 6.0)
            np.testing.assert_array_equal(a[hit].view(np.uint32), b[hit].view(np.uint32))
