"""Programmatic dependent launches, read from the sources: a kernel that is launched as a dependent may let its own successor
start only after it has waited for its predecessor.  Otherwise "the kernel before me has started" would not imply that
everything before it is complete, which is what a GEMM told that its weight is static fetches that weight on."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dsl_tool_b200", "csrc")
RELEASE, WAIT = "griddep_launch_dependents();", "griddep_wait();"


def _functions(text):
    """Bodies of the functions at namespace level: from a line that ends in `{` at column 0 to the `}` at column 0."""
    return re.findall(r"^[^\s/#}][^\n]*(?:\n[^\n{}]+)*?\{\n(.*?)^\}", text, re.S | re.M)


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "ptx.cuh"))
def test_release_comes_after_the_wait(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    bodies = [b for b in _functions(text.replace("namespace dsl {\n", "").replace("namespace {\n", "")) if RELEASE in b]
    assert sum(b.count(RELEASE) for b in bodies) == text.count(RELEASE)          # every one was seen
    for body in bodies:
        if WAIT in body:
            assert body.index(WAIT) < body.index(RELEASE)
        else:                                                                    # then it is never launched as a dependent
            assert "ProgrammaticStreamSerialization" not in text
