"""The persistent ICP's rows on the CPU (dynamap_b200/csrc/icp.cuh): a level's
rows are not overwritten by a later level, also where that level has fewer tiles
than the one before, so that blocks leave between them."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("rows") / "icp_rows.so")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared",
                    "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "cpp", "icp_rows_host.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def level_px(rows, cols, scales):
    return (C.c_int * 3)(*[(rows // s) * (cols // s) for s in scales])


def test_every_row_is_its_own(lib):
    assert lib.icp_rows_in_scratch()


def test_tiles_can_fall_from_a_level_to_the_next(lib):
    """The premise: a finer level may have fewer tiles."""
    assert lib.icp_tiles_of(330 * 248, 0) == 160 and lib.icp_tiles_of(661 * 497, 0) == 129


@pytest.mark.parametrize("kahan", [0, 1])
@pytest.mark.parametrize("scales", [(4, 2, 1), (1, 2, 4), (2, 4, 1), (2, 1, 4), (8, 4, 2),
                                    (1, 1, 1)])
def test_no_level_overwrites_rows_of_another(lib, scales, kahan):
    left = 0
    n = C.c_int(0)
    for rows in list(range(24, 760, 7)) + [497, 480, 720]:
        for cols in (rows * 4 // 3, rows * 16 // 9 + 1, 661):
            for iters in ((9, 4, 3), (2, 2, 2), (1, 3, 19), (4, 0, 2), (3, 2, 2)):
                px = level_px(rows, cols, scales)
                assert lib.icp_rows_overwritten(px, (C.c_int * 3)(*iters), kahan, C.byref(n)) == 0
                left += n.value
    if scales[0] < scales[2]:
        assert left > 0


def test_rows_are_empty_when_the_epochs_start_again(lib):
    """Tags repeat after 2^20 launches: no row of the round before survives that."""
    f = lib.icp_next_epoch
    f.restype, f.argtypes = C.c_uint, [C.c_uint, C.c_int, C.c_void_p, C.c_void_p]
    rows, before = C.c_int64(0), C.c_int64(0)
    row_bytes = (6 * 160 + 3) * 512
    for epoch in (4096, 8192, 0x7ffff000, 0xffffe000):
        assert f(epoch, 0xab, C.byref(rows), C.byref(before)) == epoch + 4096
        assert rows.value == row_bytes
    assert f(0xfffff000, 0xab, C.byref(rows), C.byref(before)) == 4096
    assert rows.value == 0 and before.value >= 160 * 29 * 8
