"""The explicit step's kernel (csrc/fs_explicit.cu, k_cd_step) may start while the
step before still writes the state and the displacement copy.  So the source must
read neither before the wait for that step, and must not tell the compiler that
the copy is read-only for the kernel's life (restrict, read-only loads)."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "finetoolsflexstructures.jl_gb300", "csrc", "fs_explicit.cu")


def _code():
    s = open(SRC).read()
    return re.sub(r"//[^\n]*", "", s)


def _function(code, name):
    """(parameters, body) of the function's definition."""
    at = re.search(r"\b%s\(" % name, code)
    i = at.end()
    depth = 1
    while depth:
        depth += {"(": 1, ")": -1}.get(code[i], 0)
        i += 1
    params = code[at.end():i - 1]
    j = code.index("{", i)
    k, depth = j + 1, 1
    while depth:
        depth += {"{": 1, "}": -1}.get(code[k], 0)
        k += 1
    return params, code[j + 1:k - 1]


def test_the_displacement_copy_is_not_declared_read_only():
    params, body = _function(_code(), "k_cd_step")
    assert re.search(r"\bxp\b", params) and re.search(r"\bxn\b", params)
    assert "__restrict__" not in params
    assert not re.search(r"__ld\w+\([^;]*\bxp\b", body)
    for m in re.finditer(r"void load6\([^{]*\{([^}]*)\}", _code()):
        assert "__ldg" not in m.group(1)


def test_nothing_of_the_step_before_is_read_before_the_wait():
    _, body = _function(_code(), "k_cd_step")
    wait = body.index("cudaGridDependencySynchronize()")
    before, after = body[:wait], body[wait:]
    for name in (r"\bxp\b", r"\bxn\b", r"\bld\b", r"s\.U\b", r"s\.cU\b", r"s\.V\b", r"s\.cV\b", r"s\.A\b"):
        assert not re.search(name, before), name
        assert re.search(name, after), name
    assert after.index("cudaTriggerProgrammaticLaunchCompletion()") > 0
