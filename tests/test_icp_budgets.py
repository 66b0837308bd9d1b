"""The shares of the device that a batch's groups take for their persistent ICP
(icp_group_budgets, dynamap_b200/csrc/icp.cuh), on the CPU: all launches fit on
the device together, for the library's own mixes and random ones; and the parts
that a table of more sessions than blocks is run in (icp_launches)."""
import ctypes as C
import os
import random
import subprocess

import pytest

from dynamap_b200 import configs

HERE = os.path.dirname(os.path.abspath(__file__))
CAP = 148  # a 512-thread block per SM


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("budgets") / "icp_rows.so")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared",
                    "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "cpp", "icp_rows_host.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.icp_weight_of.restype = C.c_longlong
    return lib


def budgets(lib, weights, counts, cap):
    k = len(weights)
    out = (C.c_int * k)()
    lib.icp_budgets((C.c_longlong * k)(*weights), (C.c_int * k)(*counts), k, cap, out)
    return list(out)


def groups(px):
    """The runs of a batch's members, largest first (dyn_batch_create)."""
    px = sorted(px, reverse=True)
    n, k = len(px), max(1, min(8, len(px) // 4))
    start, acc, g = [0] + [n] * k, 0, 1
    for j in range(n):
        if g >= k:
            break
        acc += px[j]
        if acc >= sum(px) * g / k and j + 1 <= n - (k - g):
            start[g] = j + 1
            g += 1
    for g in range(g, k):
        start[g] = max(start[g - 1] + 1, n - (k - g))
    return [px[a:b] for a, b in zip(start, start[1:])]


def check(lib, weights, counts, cap):
    b = budgets(lib, weights, counts, cap)
    assert sum(b) <= max(cap, 0)
    if sum(counts) <= cap:
        assert all(x >= c for x, c in zip(b, counts))
        plain = [cap * w // sum(weights) for w in weights]
        if all(x >= c for x, c in zip(plain, counts)):
            assert b == plain  # in proportion where that gives everyone a block
    return b


@pytest.mark.parametrize("kahan", [0, 1])
@pytest.mark.parametrize("n", [4, 17, 32, 64, 96, 128, 148, 149, 200, 400])
def test_own_mixes_fit_the_device(lib, n, kahan):
    gs = groups([p["sensor"]["rows"] * p["sensor"]["cols"] for _, p, _ in configs.session_mix(n)])
    weights = [sum(lib.icp_weight_of(x, kahan) for x in g) for g in gs]
    check(lib, weights, [len(g) for g in gs], CAP)


def test_random_groups(lib):
    rng = random.Random(5)
    for _ in range(3000):
        k = rng.randint(1, 8)
        counts = [rng.choice([1, 1, 2, 3, 5, 9, 20, 40]) for _ in range(k)]
        weights = [c * rng.choice([1000, 19200, 76800, 307200, 2764800]) for c in counts]
        check(lib, weights, counts, rng.choice([0, 1, 8, 64, 148, 132, 296]))


def test_small_groups_are_given_a_block_per_session(lib):
    assert budgets(lib, [1000000, 10], [1, 20], 148) == [128, 20]
    assert budgets(lib, [1000000, 10], [1, 200], 148) == [147, 0]  # chained kernels
    assert budgets(lib, [10, 10], [100, 100], 148) == [74, 74]     # in parts of a table
    assert budgets(lib, [5, 5], [1, 1], 0) == [0, 0]


@pytest.mark.parametrize("budget", [1, 7, 18, 74, 148, 296])
def test_parts_of_a_table(lib, budget):
    """Every launch has a block per session and fits the budget; a table is split
    only where it has to be."""
    rng = random.Random(budget)
    lib.icp_table.restype = C.c_int
    for n in list(range(1, 30)) + [37, 74, 80, 147, 148, 149, 160, 280, 296, 297, 400, 592, 700]:
        for kinds in (lambda: 0, lambda: 1, lambda: rng.randint(0, 1)):
            for sizes in ([3072], [19200], [3072, 19200, 307200]):
                px = [rng.choice(sizes) for _ in range(n)]
                kahan = [kinds() for _ in range(n)]
                grid, first = (C.c_int * 8)(), (C.c_int * 5)()
                parts = lib.icp_table((C.c_int * n)(*px), (C.c_int * n)(*kahan), n, budget, grid, first)
                assert parts == (0 if n > 4 * budget else -(-n // budget))
                if parts == 0:
                    continue
                assert first[0] == 0 and first[parts] == n
                for p in range(parts):
                    for kind in (0, 1):
                        members = sum(k == kind for k in kahan[first[p]:first[p + 1]])
                        assert members <= grid[2 * p + kind] <= budget
                        assert (grid[2 * p + kind] == 0) == (members == 0)
