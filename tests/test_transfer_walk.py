"""The walk of the batch transfer kernels over a grid's words and 16-cell vectors,
compiled for the host from the kernels' own header: every item once, on grids whose
items are counted past 2^31 too."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STRIDE = 16 * 256  # threads on one grid


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("transfer") / "transfer.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "cat_cpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "transfer_walk_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.row_walk_host.restype = ctypes.c_longlong
    return lib


def walk(host, at, stride, width, rows):
    total, last = ctypes.c_ulonglong(), ctypes.c_longlong()
    count = host.row_walk_host(at, stride, width, rows, ctypes.byref(total), ctypes.byref(last))
    return count, total.value, last.value


@pytest.mark.parametrize("n", [1, 5, 31, 32, 33, 63, 64, 65, 2048, 185351, 185352, 200000, 262143, 262144, 379000])
def test_items_of_a_grid(host, n):
    for width in ((n + 31) // 32, (n + 15) // 16 + 1):  # words, vectors
        items = n * width
        for at in (0, 1, STRIDE // 2 + 7, STRIDE - 1):
            count = max(0, -(-(items - at) // STRIDE))
            last = at + (count - 1) * STRIDE
            want = (count, (count * (at + last) // 2) % 2**64 if count else 0, last if count else -1)
            assert walk(host, at, STRIDE, width, n) == want, (n, width, at)
