"""Kernels are resident while the kernels before them on the stream still write
their inputs (they wait in dependent_start, common.cuh).  What that asks of the
sources is checked here, on the text: every kernel waits first, no load takes
the read-only path, and no input parameter is declared unaliased."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ochre_gb300", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _code(path):
    """The source without its comments."""
    with open(path) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _after(text, open_at):
    """Index just past the bracket that closes the one at open_at."""
    close = {"(": ")", "{": "}"}[text[open_at]]
    depth = 0
    for i in range(open_at, len(text)):
        depth += (text[i] == text[open_at]) - (text[i] == close)
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_kernels_wait_first_and_read_by_ordinary_loads(path):
    text = _code(path)
    assert "__ldg" not in text and "ld.global.nc" not in text
    assert not re.findall(r"const\s+[\w:<>]+\s*\*\s*__restrict__", text)
    for m in re.finditer(r"__global__", text):
        at = re.compile(r"\bvoid\b").search(text, m.end()).end()
        if "__launch_bounds__" in text[m.end():text.index("{", at)]:
            at = _after(text, text.index("(", text.index("__launch_bounds__", m.end())))
        name = re.compile(r"\bk_\w+").search(text, at)
        body = text[_after(text, text.index("(", name.end())):].lstrip()
        assert body.startswith("{") and body[1:].lstrip().startswith("dependent_start();"), name.group()
