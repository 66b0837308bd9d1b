"""Which rays may march through the block grid (dynamap_b200/csrc/ray_grid.cuh):
the march reads the grid without checks, so every block that such a ray can look
up has to lie in the grid's box, and a pose with an entry that is not finite, or
beyond the range of the indices, takes the hash.  On the CPU for every entry of
the pose; on the GPU, renders at such poses equal those of a session without a
grid."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from dynamap_b200 import abi, configs

HERE = os.path.dirname(os.path.abspath(__file__))
CAP = 1 << 24
BAD = [np.nan, np.inf, -np.inf, 3e38, -3e38, 1e20]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_fp16.h"):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("raygrid") / "raygrid.so")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared", "-ffp-contract=off",
                    "-I", "/usr/local/cuda/include", os.path.join(HERE, "cpp", "ray_grid_host.cpp"),
                    "-o", so], check=True)
    lib = C.CDLL(so)

    def run(pose, rows=48, cols=64, f=52.5, tsdf=(0.01, 0.04, 3.0), step=5, samples=40):
        pose = np.ascontiguousarray(pose, np.float32)
        sens = np.array([f, f, (cols - 1) / 2, (rows - 1) / 2], np.float32)
        ts = np.array(tsdf, np.float32)
        out = np.zeros(4, np.int64)
        lib.ray_grid_check(pose.ctypes.data_as(C.c_void_p), sens.ctypes.data_as(C.c_void_p), rows,
                           cols, ts.ctypes.data_as(C.c_void_p), CAP, step, samples,
                           out.ctypes.data_as(C.c_void_p))
        return out

    return run


def rigid(rng, reach):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    T = np.eye(4)
    T[:3, :3] = q * np.sign(np.diag(r))
    T[:3, 3] = rng.uniform(-reach, reach, 3)
    return T


@pytest.mark.parametrize("reach", [0.5, 20.0, 1200.0])
def test_rigid_poses_stay_in_the_box(check, reach):
    rng = np.random.default_rng(3)
    for _ in range(40):
        exact, mixed, outside, ok = check(rigid(rng, reach))
        assert ok and exact > 0 and mixed > 0 and outside == 0


@pytest.mark.parametrize("entry", range(12))
def test_a_pose_that_is_not_finite_takes_the_hash(check, entry):
    rng = np.random.default_rng(entry)
    for bad in BAD:
        T = rigid(rng, 2.0)
        T[entry // 4, entry % 4] = bad
        exact, mixed, outside, ok = check(T)
        assert exact == 0 and mixed == 0 and outside == 0 and not ok
        # the ray's own test, with a box made at another pose
        T2 = rigid(rng, 2.0)
        T2[(entry // 4 + 1) % 3, entry % 4] = bad
        T2[entry // 4, 3] = bad
        assert check(T2)[:3].sum() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [abi.PRECISION_FP32, abi.PRECISION_MIXED])
def test_renders_at_such_poses(gpu_lib, prec):
    from dynamap_b200.session import Session

    def session(dmax):
        p = configs.preset("cfg1")
        p["sensor"].update(rows=48, cols=64, fx=52.5, fy=52.5, cx=31.5, cy=23.5)
        p["tsdf"].update(num_blocks=1 << 13, num_buckets=1 << 14, voxel_size=0.02,
                         truncation_distance=0.08, max_sensor_depth=dmax)
        p["gn"].update(lvl_scale=[1, 1, 1])
        seq = configs.sequence(p, seed=5, n_frames=1)
        t, g, b, s = configs.structs(p)
        m = Session(t, g, b, s, precision=prec)
        m.integrate_with_pose(seq.depth[0], None, seq.poses[0].astype(np.float32))
        return m, seq.poses[0].astype(np.float32)

    near, pose = session(6.0)   # rays through the grid
    far, _ = session(80.0)      # too large a box: through the hash
    with near, far:
        good = near.raycast(pose)[0]
        assert (good < 6.0).any()
        for entry in range(12):
            for bad in (np.nan, np.inf):
                q = pose.copy()
                q[entry // 4, entry % 4] = bad
                a, b = near.raycast(q)[0], far.raycast(q)[0]
                hit = a < 6.0
                np.testing.assert_array_equal(hit, b < 6.0)
                np.testing.assert_array_equal(a[hit].view(np.uint32), b[hit].view(np.uint32))
        np.testing.assert_array_equal(near.raycast(pose)[0], good)
