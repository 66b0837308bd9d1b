"""The chained ICP (a launch per iteration) and the persistent one (one launch
per frame) give the same bits: tables of both summation kinds with different
iteration counts, and sessions whose levels differ in the shape of their tiles."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from dynamap_b200 import abi

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Runs in a child process: the chained form is chosen when the library loads
# (DYN_ICP_CHAINED).  argv: root, output file, tables; a table of one member is
# a session, one of more a batch.
CHILD = r"""
import json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from dynamap_b200 import configs
from dynamap_b200.session import Session, Batch
out = []
for table in json.loads(sys.argv[3]):
    ss, seqs = [], []
    for j, m in enumerate(table):
        p = configs.preset("cfg2" if m["rgb"] else "cfg1")
        f = 525.0 * m["cols"] / 640.0
        p["sensor"].update(rows=m["rows"], cols=m["cols"], fx=f, fy=f, cx=(m["cols"] - 1) / 2.0,
                           cy=(m["rows"] - 1) / 2.0)
        p["tsdf"].update(num_blocks=1 << 14, num_buckets=1 << 15, voxel_size=0.02,
                         truncation_distance=0.08)
        p["gn"].update(lvl_scale=m["scales"], lvl_iteration_num=m["iters"])
        seqs.append(configs.sequence(p, seed=60 + j, n_frames=4))
        t, g, b, s = configs.structs(p)
        ss.append(Session(t, g, b, s, precision=m["prec"]))
        ss[-1].set_pose(seqs[-1].poses[0])
    rgb = lambda m, q, k: q.rgb[k] if m["rgb"] else None
    for k in range(4):
        if len(ss) == 1:
            got = [ss[0].process(seqs[0].depth[k], rgb(table[0], seqs[0], k))]
        else:
            if k == 0:
                bt = Batch(ss)
            poses, stats, _ = bt.process([q.depth[k] for q in seqs],
                                         [rgb(m, q, k) for m, q in zip(table, seqs)])
            got = list(zip(poses, stats))
        for pose, st in got:
            out.append(np.concatenate([pose.reshape(16), np.array(st.icp_iterations, np.float32),
                                       np.array(st.icp_inliers, np.float32)]))
    if len(ss) > 1:
        bt.close()
    for s in ss:
        s.close()
np.save(sys.argv[2], np.array(out, np.float32))
"""


def member(rows, cols, prec, iters, scales=(4, 2, 1), rgb=False):
    return dict(rows=rows, cols=cols, prec=prec, iters=list(iters), scales=list(scales), rgb=rgb)


def run_form(tmp_path, tables, chained):
    out = str(tmp_path / f"rows_{int(chained)}.npy")
    env = dict(os.environ)
    env.pop("DYN_ICP_CHAINED", None)
    if chained:
        env["DYN_ICP_CHAINED"] = "1"
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, out, json.dumps(tables)], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return np.load(out)


def assert_forms_agree(tmp_path, tables):
    a, b = run_form(tmp_path, tables, False), run_form(tmp_path, tables, True)
    assert a.shape == b.shape and len(a) == 4 * sum(len(t) for t in tables)
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
    assert (a[:, 16:19].max(axis=1) > 0).sum() >= len(a) * 3 // 4  # all but the first frames


def test_kinds_of_different_iteration_counts(tmp_path, gpu_lib):
    """A launch without work for any session of its kind stands between two
    launches of the other kind."""
    few, many = (3, 2, 2), (10, 5, 4)
    fp32, mixed = abi.PRECISION_FP32, abi.PRECISION_MIXED
    assert_forms_agree(tmp_path, [
        [member(120, 160, fp32, few), member(120, 160, mixed, many)],
        [member(120, 160, fp32, many), member(120, 160, mixed, few),
         member(96, 128, mixed, many, rgb=True)]])


FP32, MIXED = abi.PRECISION_FP32, abi.PRECISION_MIXED


def test_tile_shapes(tmp_path, gpu_lib):
    """Levels where the tiles change shape: a level of 256-slot tiles at its
    largest and one pixel row beyond, blocks that leave before the last level
    (more tiles on a coarser level, levels from fine to coarse), pixel groups of
    one, two and four in the compensated form, ragged levels."""
    it = (5, 4, 4)
    tables = [member(497, 661, FP32, it),                   # 41, 160, 129 tiles
              member(148, 256, FP32, it), member(149, 256, FP32, it), member(147, 257, FP32, it),
              member(120, 160, FP32, it, (1, 2, 4)), member(497, 661, FP32, it, (1, 2, 4)),
              member(120, 160, MIXED, it, (1, 2, 4), rgb=True), member(240, 320, FP32, it, (2, 4, 1)),
              member(64, 128, MIXED, it), member(65, 127, MIXED, it),
              member(256, 256, MIXED, it), member(257, 255, MIXED, it, rgb=True),
              member(133, 177, FP32, it, rgb=True), member(133, 177, MIXED, it, (8, 4, 1)),
              member(24, 40, FP32, it, (8, 2, 1)), member(24, 40, MIXED, it, (8, 2, 1))]
    assert_forms_agree(tmp_path, [[m] for m in tables])


def test_batches_of_many_sessions(tmp_path, gpu_lib):
    """More sessions than a group's part of the device has blocks: 66 members of
    three sizes and both kinds, their groups' launches running at once."""
    it = (4, 3, 3)
    sizes = [(48, 64), (48, 64), (48, 64), (120, 160), (48, 64), (240, 320)]
    assert_forms_agree(tmp_path, [[member(*sizes[i % 6], (FP32, MIXED)[i % 4 == 1], it)
                                   for i in range(66)]])


def test_tables_in_parts(tmp_path, gpu_lib):
    """More sessions than the device has resident blocks: the persistent form runs
    the table in parts."""
    it = (4, 3, 3)
    assert_forms_agree(tmp_path, [[member(32, 48, (FP32, MIXED)[i % 3 == 1], it)
                                   for i in range(170)]])
