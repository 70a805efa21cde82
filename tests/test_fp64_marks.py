"""When marked elements are done over in double (FxMarks of csrc/fs_fp64_rows.h on
the host): only after element kernels that wrote the marks, not after others that
find the device's flag still set by a call which failed before it was read; and
in the sources, every element launch starts anew."""
import ctypes
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "finetoolsflexstructures.jl_gb300", "csrc")


@pytest.mark.parametrize("events,redos", [
    ("lmR", 1),        # marked elements
    ("lmr", 0),        # none marked
    ("lmlmR", 1),      # the tuner's launches
    ("lmlR", 0),       # failed before the read; then a mixed, layered or beam assembly
    ("lmrlR", 0),
    ("lmRlR", 1),      # once
    ("lmlRlmR", 1),   # a later FP64 call has its own
    ("R", 0),
])
def test_marks_of_the_last_launch(tmp_path, events, redos):
    so = str(tmp_path / "librowscheck.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    os.path.join(HERE, "hostcheck", "rowscheck.cpp")], check=True)
    assert ctypes.CDLL(so).marks_events(events.encode()) == redos


@pytest.mark.parametrize("file,name", [("fs_numeric.cu", "launch_elements"), ("fs_numeric.cu", "launch_elements_to"),
                                       ("fs_beam.cu", "launch_beam_elements")])
def test_every_element_launch_starts_anew(file, name):
    s = open(os.path.join(CSRC, file)).read()
    body = re.search(r"^int %s\([^)]*\)\n\{\n(.*?)^\}" % name, s, re.S | re.M).group(1)
    assert body.strip().startswith("c->fx_marks.launch();")


def test_the_flag_alone_does_not_decide():
    s = open(os.path.join(CSRC, "fs_elem_fp64.cu")).read()
    body = re.search(r"^int read_element_status\([^)]*\)\n\{\n(.*?)^\}", s, re.S | re.M).group(1)
    assert "c->fx_marks.redo(" in body
    assert body.index("fx_marks.redo(") < body.index("redo_t3(")
