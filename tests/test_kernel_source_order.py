"""Orders that a race would hide behind on every machine at hand, read off the kernels' source (no GPU)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _body(name, unit):
    """The text of a function's body, comments taken out."""
    text = open(os.path.join(ROOT, "heatflow_gb300", "csrc", unit)).read()
    text = re.sub(r"//[^\n]*", "", text)
    at = text.index("{", re.search(rf"\b{name}\(", text).end())
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[at:k + 1]
    raise AssertionError(name)


def test_finalize_reads_flags_before_the_epilogue_writes_them():
    """All threads of k_finalize read the shared scalars' flags, then one thread's epilogue rewrites them:
    a block barrier lies between, or a late warp would not write its words back."""
    body = _body("k_finalize", "hf_solve.cu")
    read, write = body.index("took_part<KIND>(sh)"), body.index("epi_rhs(sh")
    assert read < write
    assert "__syncthreads()" in body[read:write]


def test_warp_votes_name_lanes_that_arrive():
    """A vote over __activemask() names whichever lanes happen to run together and then waits for them:
    the kernels vote with all lanes, which take the same number of rounds."""
    for unit in os.listdir(os.path.join(ROOT, "heatflow_gb300", "csrc")):
        text = open(os.path.join(ROOT, "heatflow_gb300", "csrc", unit)).read()
        assert "__activemask" not in text, unit


def test_refused_instantiation_leaves_no_handle():
    """A graph whose instantiation is refused has no executable: every instantiation goes through the one
    place that says so, and none of the error paths destroys what was never made."""
    text = open(os.path.join(ROOT, "heatflow_gb300", "csrc", "hf_abi.cu")).read()
    assert text.count("cudaGraphInstantiate(") == 1
    assert "nullptr" in _body("instantiate", "hf_abi.cu")
