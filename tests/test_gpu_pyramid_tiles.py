"""Pyramid and normals of a frame's source and target at the edges of the
kernel's 32x16 tiles: images smaller than a tile, a pixel off its multiples, odd
sizes whose upper levels drop a row or column, one to four levels, with colours
and without, frame-to-model and frame-to-frame, holes in the depth.  Bit for bit
the oracle's levels of the same level 0."""
import numpy as np
import pytest

from dynamap_b200 import configs
from dynamap_b200.session import Session

pytestmark = pytest.mark.gpu


SIZES = [(16, 32), (17, 33), (15, 31), (41, 70), (66, 131)]
FORMS = [((1, 1, 1), 1, 1.0), ((1, 2, 4), 1, 0.0), ((1, 2, 4), 0, 1.0), ((1, 4, 8), 1, 1.0)]


# a session refuses a level below 3 rows or 5 columns
@pytest.mark.parametrize("rows,cols,scale,mode,colour",
                         [z + f for z in SIZES for f in FORMS
                          if z[0] // f[0][2] >= 3 and z[1] // f[0][2] >= 5])
def test_levels_match_oracle(gpu_lib, oracle, rows, cols, scale, mode, colour):
    p = configs.preset("cfg2")
    fx = 525.0 * cols / 640.0
    p["sensor"].update(rows=rows, cols=cols, fx=fx, fy=fx, cx=(cols - 1) / 2, cy=(rows - 1) / 2)
    p["tsdf"].update(num_blocks=1 << 12, num_buckets=1 << 13, voxel_size=0.02,
                     truncation_distance=0.08)
    p["gn"].update(lvl_scale=list(scale), mode=mode, color_weight=colour)
    seq = configs.sequence(p, seed=5, n_frames=1)
    rng = np.random.default_rng(rows * cols)
    depth = np.where(rng.random((rows, cols)) < 0.05, 0, seq.depth[0]).astype(np.uint16)
    t, g, b, s = configs.structs(p)

    def same(a, r):
        np.testing.assert_array_equal(a.view(np.uint32), np.asarray(r).view(np.uint32))

    with Session(t, g, b, s) as m:
        m.set_pose(seq.poses[0])
        m.process(depth, seq.rgb[0] if colour else None)
        shape = (rows, cols)
        for dep, vtx, nrm, ints in ((2, 3, 4, 9), (5, 6, 7, 10)):
            d = m.image(dep, 0, shape, np.float32)
            assert np.any(d > 0)
            if dep == 2:
                same(d, m.image(1, 0, shape, np.float32))
            elif mode == 0:
                same(d, m.image(2, 0, shape, np.float32))
            i = m.image(ints, 0, shape, np.float32) if colour else None
            if colour and dep == 2:
                same(i, oracle.intensity(seq.rgb[0]))
            for l in range(max(scale).bit_length()):
                sh = (rows >> l, cols >> l)
                if l:
                    d = oracle.downsample_depth(d)
                    same(m.image(dep, l, sh, np.float32), d)
                    if colour:
                        i = oracle.downsample_intensity(i)
                        same(m.image(ints, l, sh, np.float32), i)
                v, n = oracle.maps(d, oracle.level_sensor(s, 1 << l))
                same(m.image(nrm, l, sh + (4,), np.float32), n)
                same(m.image(vtx, l, sh + (4,), np.float32), v)
