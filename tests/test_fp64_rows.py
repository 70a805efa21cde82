"""Sizes of the FS_FP64 elements' row buffer (csrc/fs_fp64_rows.h on the host) in
a memory that may be too small: what a chunk takes lies within the buffer, a chunk
is never empty while there is a buffer, and a buffer that came out small is
neither asked for by every assembly nor kept for the next mesh."""
import ctypes
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LEAST = 608


class Rows(ctypes.Structure):
    _fields_ = [("cap", ctypes.c_uint64), ("asked", ctypes.c_uint64), ("tries", ctypes.c_uint64)]


@pytest.fixture(scope="module")
def reserve(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rows") / "librowscheck.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "finetoolsflexstructures.jl_gb300", "csrc"),
                    "-o", so, os.path.join(HERE, "hostcheck", "rowscheck.cpp")], check=True)
    f = ctypes.CDLL(so).rows_reserve
    f.restype = ctypes.c_uint64
    f.argtypes = [ctypes.POINTER(Rows)] + [ctypes.c_uint64] * 4

    def call(r, nelem, memory, group=32 * 129):
        """The groups of a chunk and the mesh's (marks, groups a chunk asks for)."""
        groups, most = (nelem + 31) // 32, (1 << 27) // group
        chunks = max((groups + most - 1) // most, 1)
        marks, want = (nelem + 255) // 256 * 32, max((groups + chunks - 1) // chunks, 1)
        return f(ctypes.byref(r), marks, want, group, memory), marks, want
    return call


def check(r, got, marks, want, group=32 * 129):
    assert got <= want
    if r.cap == 0:
        assert got == 0
    else:
        assert got >= min(want, LEAST) and marks + got * group <= r.cap


def test_a_small_buffer_is_not_taken_for_a_large_mesh(reserve):
    # 1 M triangles get the smallest chunk; 20 M in the same memory need more than
    # that for their marks alone
    r = Rows()
    memory = 3 * (1 << 20)
    got, marks, want = reserve(r, 1 << 20, memory)
    check(r, got, marks, want)
    assert 0 < got < want
    got, marks, want = reserve(r, 20 << 20, memory)
    check(r, got, marks, want)


def test_marks_that_just_fit_leave_no_empty_chunk(reserve):
    r = Rows()
    reserve(r, 1 << 20, 3 * (1 << 20))
    for nelem in range(r.cap // 32 * 256 - 4096, r.cap // 32 * 256 + 4096, 256):
        s = Rows(r.cap, r.asked, 0)
        got, marks, want = reserve(s, nelem, 1 << 40)
        check(s, got, marks, want)
        assert got > 0


def test_one_search_a_mesh(reserve):
    r = Rows()
    memory = 4 * (1 << 20)
    got = reserve(r, 1 << 20, memory)[0]
    tries = r.tries
    for _ in range(5):
        assert reserve(r, 1 << 20, memory)[0] == got
    assert r.tries == tries
    r.asked = 0  # a new mesh, and memory again
    got, marks, want = reserve(r, 1 << 20, 1 << 40)
    assert got == want
    tries = r.tries
    assert reserve(r, 1 << 19, 0)[0] > 0 and r.tries == tries   # a smaller mesh fits what is there


def test_any_sequence(reserve):
    rng = random.Random(5)
    for _ in range(300):
        r = Rows()
        for _ in range(8):
            nelem = int(2 ** rng.uniform(0, 28))
            group = 32 * rng.choice([129, 130, 350])
            if rng.random() < 0.5:
                r.asked = 0
            got, marks, want = reserve(r, nelem, int(2 ** rng.uniform(8, 30)), group)
            check(r, got, marks, want, group)
