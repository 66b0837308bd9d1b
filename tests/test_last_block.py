"""The ticket by which the ICP's reductions find their last block
(dynamap_b200/csrc/last_block.cuh), run on the CPU: a block's ticket waits for
the stores of all its threads, and one block is told to be the last."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_fp16.h"):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("last") / "last_block.so")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared",
                    "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "cpp", "last_block_host.cpp"), "-o", so], check=True)
    return C.CDLL(so).last_block_check


# (the chained kernel's and the stage kernel's shapes, a value per thread, one block)
@pytest.mark.parametrize("blocks,threads,values", [(75, 512, 29), (9, 256, 29), (3, 64, 64),
                                                   (1, 512, 29)])
def test_ticket_waits_for_the_blocks_stores(check, blocks, threads, values):
    last = C.c_int(0)
    assert check(blocks, threads, values, C.byref(last)) == 0
    assert last.value == 1
