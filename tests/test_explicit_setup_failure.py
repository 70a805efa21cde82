"""A failed fs_explicit_setup leaves no explicit state behind: buffers that it could
not allocate are gone, so a run on an earlier set-up's word would read nothing.
On the source, since the failure is an exhausted device: the state ends before the
first buffer is replaced, and is declared ready at the very end."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "finetoolsflexstructures.jl_gb300", "csrc", "fs_explicit.cu")


def test_no_state_while_setting_up():
    s = re.sub(r"//[^\n]*", "", open(SRC).read())
    end = re.search(r"void end_explicit\(fs_ctx \*c\)\n\{\n(.*?)^\}", s, re.S | re.M).group(1)
    assert "x.ready = false;" in end
    body = re.search(r"int fs_explicit_setup\([^)]*\)\n\{\n(.*?)^\}", s, re.S | re.M).group(1)
    first = min(body.index(w) for w in ("dalloc(", "cudaMalloc(", "dfree("))
    assert "end_explicit(c);" in body[:first]
    ready = body.index("x.ready = true;")
    assert "return" in body[ready:] and not re.search(r"FS_(TRY|CUDA)\(", body[ready:])
    # errors of the arguments are refused before that, and keep the state
    assert body.index("time step must be positive") < body.index("end_explicit(c);")
