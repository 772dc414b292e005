"""The registry of pinned host ranges: how much of an array the GPU reaches through a range, compiled on its own."""
import ctypes as C
import os
import subprocess

SRC = r"""
#include "pinned.h"
static mdg::PinnedRanges ranges;
extern "C" void add(size_t p, size_t n, size_t dev) { ranges.add((void*)p, n, (void*)dev); }
extern "C" void drop(size_t p) { ranges.remove((void*)p); }
extern "C" size_t find(size_t p, size_t n, size_t* room) { return (size_t)ranges.find((void*)p, n, *room); }
"""


def test_ranges(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "t.cpp").write_text(SRC)
    out = tmp_path / "t.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(root, "md_sim_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    for f in (lib.add, lib.drop, lib.find):
        f.argtypes = [C.c_size_t] * (1 if f is lib.drop else 3) if f is not lib.find else [C.c_size_t, C.c_size_t, C.POINTER(C.c_size_t)]
    lib.find.restype = C.c_size_t

    def find(p, n):
        room = C.c_size_t(99)
        return lib.find(p, n, C.byref(room)), room.value

    assert find(4096, 8) == (0, 0)
    lib.add(4096, 1000, 70000)
    lib.add(8192, 4096, 90000)
    assert find(4096, 1000) == (70000, 1000)   # the whole range
    assert find(4196, 900) == (70100, 900)     # up to its end
    assert find(4196, 901) == (70100, 900)     # beyond it: only what is pinned
    assert find(5092, 64) == (70996, 4)        # a word that straddles the end
    assert find(5096, 8) == (0, 0) and find(4000, 200) == (0, 0)  # from the end, and from before the start
    assert find(8192 + 4088, 16) == (90000 + 4088, 8)
    lib.drop(4096)
    assert find(4196, 8) == (0, 0) and find(9000, 8) == (90808, 8)
