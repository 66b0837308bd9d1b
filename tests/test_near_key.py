"""Allocation's tile-local block keys (dynamap_b200/csrc/near_key.cuh) on the
CPU: a walk that is taken with them names the blocks that it steps through, at
the ends of the fields too, and one that could leave the fields is refused, at
the ends of the integers too."""
import ctypes as C
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
BIG = 2 ** 31 - 1


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_fp16.h"):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("near") / "near_key.so")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared",
                    "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "cpp", "near_key_host.cpp"), "-o", so], check=True)
    f = C.CDLL(so).near_walk_check

    def run(wide, o, left, axis=0, s=1, cam=(0, 0, 0)):
        return f(wide, (C.c_int * 3)(*o), (C.c_int * 3)(*cam), left, axis, s)

    return run


@pytest.mark.parametrize("wide,half", [(0, 512), (1, 1 << 20)])
def test_ends_of_the_fields(check, wide, half):
    for left in (0, 1, 300):
        edge = half - 2 - left  # the farthest start
        for axis in range(3):
            for s in (1, -1):
                for start in (edge, -edge, 0):
                    o = [0, 0, 0]
                    o[axis] = start
                    assert check(wide, o, left, axis, s) == 0
                    o[axis] = start + (1 if start >= 0 else -1) if start else half - 1 - left
                    assert check(wide, o, left, axis, s) == -1


@pytest.mark.parametrize("wide", [0, 1])
def test_ends_of_the_integers_are_refused(check, wide):
    for v in (BIG, BIG - 1, BIG - 300, -BIG - 1, -BIG, -BIG + 300, 1 << 30, -(1 << 30), 1 << 21):
        for axis in range(3):
            for left in (0, 1, 8, 300, 509, BIG):
                o = [0, 0, 0]
                o[axis] = v
                assert check(wide, o, left, axis) == -1
    assert check(wide, (0, 0, 0), BIG) == -1


@pytest.mark.parametrize("wide,half", [(0, 512), (1, 1 << 20)])
def test_random_walks(check, wide, half):
    rng = random.Random(1)
    taken = 0
    for _ in range(3000):
        o = [rng.randint(-half, half) // rng.choice([1, 2, 8]) for _ in range(3)]
        cam = [rng.randint(-90000, 90000) for _ in range(3)]
        r = check(wide, o, rng.randint(0, min(half, 900)) // rng.choice([1, 3]), rng.randint(0, 2),
                  rng.choice([1, -1]), cam)
        assert r in (-1, 0)
        taken += r == 0
    assert taken > 300
