"""Every wait in a kernel has a limit, which the launch gives it: a wait without one hangs the GPU for everybody where what it waits for
does not come.  Shown by reading the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ac4k_kernel_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def _arguments(text, at):
    """the arguments of the call whose opening parenthesis is text[at]"""
    depth, args, start = 0, [], at + 1
    for i in range(at, len(text)):
        depth += text[i] in "([{"
        depth -= text[i] in ")]}"
        if depth == 0 or (depth == 1 and text[i] == ","):
            args.append(text[start:i].strip())
            start = i + 1
        if depth == 0:
            return args


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_waits_carry_the_limit_of_the_launch(path):
    text = _code(path)
    for call in re.finditer(r"(?<!bool )\bmbar_wait\(", text):
        args = _arguments(text, call.end() - 1)
        assert len(args) == 3 and args[2].endswith("wait_ns"), args


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_grid_barrier_without_a_limit(path):
    assert not re.search(r"cooperative_groups|this_grid\(|grid_group", _code(path))
