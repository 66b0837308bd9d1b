"""The blocks that a frame allocates, in each form of the rays' sets: 10-bit
offsets from the camera's block (few steps a ray), 21-bit ones (small voxels),
rays from the camera and from the surface band, more blocks a tile than its set
holds, cameras far from the origin on either side, and a pose that is not rigid
(starts beyond 10 bits).  The same blocks as the oracle's walk of every ray,
with the points in the reference's FP32 operations."""
import numpy as np
import pytest

from dynamap_b200 import abi, configs
from dynamap_b200.session import Batch, Session

pytestmark = pytest.mark.gpu
F = np.float32


def expected(oracle, d, s, t, T, band):
    bs = F(8) * F(t.voxel_size)
    cap = 3 * int(np.ceil((t.max_sensor_depth + t.truncation_distance) / float(bs))) + 8
    cam, out = T[:3, 3], set()
    for y in range(s.rows):
        for x in range(s.cols):
            z = d[y, x]
            if z < F(t.min_sensor_depth) or z > F(t.max_sensor_depth):
                continue
            p = ((F(x) - F(s.cx)) * z / F(s.fx), (F(y) - F(s.cy)) * z / F(s.fy), z)
            w = np.array([((T[r, 0] * p[0] + T[r, 1] * p[1]) + T[r, 2] * p[2]) + T[r, 3]
                          for r in range(3)], F)
            st = cam
            if band:
                v = w - cam
                inv = F(1) / np.sqrt((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2])
                st = w - (v * inv) * F(t.truncation_distance)
            blocks, ok = oracle.dda_blocks(st, w, t.truncation_distance, float(bs), cap)
            assert ok
            out.update(map(tuple, blocks))
    return out


@pytest.mark.parametrize("band", [False, True])
@pytest.mark.parametrize("voxel,scale,shift", [(0.02, 1, 0.0), (0.02, 1, -40.0), (0.004, 1, 3.0),
                                               (0.004, 4, 0.5), (0.003, 1, -1.0), (0.002, 1, 0.0)])
def test_allocated_blocks(gpu_lib, oracle, voxel, scale, shift, band):
    if scale != 1 and not band:
        pytest.skip("a ray from the camera may not outrun its cap")
    p = configs.preset("cfg1")
    rows, cols = 18, 25
    fx = 525.0 * cols / 640.0
    p["sensor"].update(rows=rows, cols=cols, fx=fx, fy=fx, cx=(cols - 1) / 2, cy=(rows - 1) / 2)
    p["tsdf"].update(num_blocks=1 << 17, num_buckets=1 << 18, voxel_size=voxel,
                     truncation_distance=4 * voxel, max_sensor_depth=3.0)
    p["gn"].update(lvl_scale=[1, 1, 1])
    seq = configs.sequence(p, seed=9, n_frames=1)
    t, g, b, s = configs.structs(p)
    T = seq.poses[0].astype(F)
    T[:3, :3] *= F(scale)
    T[:3, 3] += F(shift)
    with Session(t, g, b, s,
                 precision=abi.PRECISION_MIXED_BAND if band else abi.PRECISION_FP32) as m:
        m.integrate_with_pose(seq.depth[0], None, T)
        got = {tuple(c) for c in m.download_blocks()[0]}
    ref = expected(oracle, oracle.depth_from_raw(seq.depth[0], s.depth_scaler), s, t, T, band)
    assert len(ref) > 100
    assert got == ref


def narrow_view(fx, voxel):
    p = configs.preset("cfg1")
    rows, cols = 35, 50
    p["sensor"].update(rows=rows, cols=cols, fx=fx, fy=fx, cx=(cols - 1) / 2, cy=(rows - 1) / 2)
    p["tsdf"].update(num_blocks=1 << 14, num_buckets=1 << 15, voxel_size=voxel,
                     truncation_distance=4 * voxel, max_sensor_depth=3.0)
    p["gn"].update(lvl_scale=[1, 1, 1])
    return p


@pytest.mark.parametrize("band", [False, True])
@pytest.mark.parametrize("fx", [74.0, 76.0, 150.0])
def test_close_rays(gpu_lib, oracle, fx, band):
    """Neighbouring rays in the same blocks: either side of the line of rays from
    the camera (four a block at the sensor range: fx 75 at 2 cm and 3 m)."""
    p = narrow_view(fx, 0.02)
    seq = configs.sequence(p, seed=9, n_frames=1)
    t, g, b, s = configs.structs(p)
    T = seq.poses[0].astype(F)
    with Session(t, g, b, s,
                 precision=abi.PRECISION_MIXED_BAND if band else abi.PRECISION_FP32) as m:
        m.integrate_with_pose(seq.depth[0], None, T)
        got = {tuple(c) for c in m.download_blocks()[0]}
    assert len(got) > 20
    assert got == expected(oracle, oracle.depth_from_raw(seq.depth[0], s.depth_scaler), s, t, T,
                           band)


def test_close_and_apart_in_one_table(gpu_lib):
    """A batch of both kinds: every member's blocks as alone, the next frame's
    target (its grid emptied beside the rays) as well."""
    specs = [(150.0, 0.02), (31.0, 0.02), (150.0, 0.02), (150.0, 0.004)]
    ps = [narrow_view(f, v) for f, v in specs]
    ps[3]["tsdf"].update(num_blocks=1 << 16, num_buckets=1 << 17)
    seqs = [configs.sequence(p, seed=3 + j, n_frames=3) for j, p in enumerate(ps)]

    def make(j):
        t, g, b, s = configs.structs(ps[j])
        m = Session(t, g, b, s)
        m.set_pose(seqs[j].poses[0].astype(F))
        return m

    alone = []
    for j in range(4):
        with make(j) as m:
            poses = [m.process(seqs[j].depth[k])[0] for k in range(3)]
            alone.append((np.array(poses), sorted(map(tuple, m.download_blocks()[0]))))
    ss = [make(j) for j in range(4)]
    with Batch(ss) as bt:
        got = [bt.process([q.depth[k] for q in seqs])[0] for k in range(3)]
    for j, m in enumerate(ss):
        poses, blocks = alone[j]
        for k in range(3):
            np.testing.assert_array_equal(np.asarray(got[k][j]).view(np.uint32),
                                          poses[k].view(np.uint32))
        assert sorted(map(tuple, m.download_blocks()[0])) == blocks
        m.close()
