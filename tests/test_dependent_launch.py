"""Kernels that wait for the kernel before them (pdl_wait) while that one still
writes promise nothing about their arrays: no __restrict__ pointers."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "flowlb_b200" / "csrc"
# written last by the flag pass one step back, which FS_1 between the two waited for
FINISHED = {("k_fs234", "nz")}


def closing(text, start):
    """Position of the bracket that closes the one at text[start]."""
    pair = {"(": ")", "{": "}"}[text[start]]
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == text[start]) - (text[i] == pair)
        if depth == 0:
            return i
    raise AssertionError("unbalanced source")


def dependent_kernels():
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"\b(k_\w+)\s*\(").search(text, m.end())
            end = closing(text, head.end() - 1)
            body = text.index("{", end)
            if ";" in text[end:body]:
                continue  # a declaration
            if "pdl_wait()" in text[body:closing(text, body)]:
                yield path.name, head.group(1), text[head.end():end]


def test_no_restrict_parameters():
    found = list(dependent_kernels())
    assert {"k_por_fwd", "k_por_bwd", "k_fs1", "k_fs234", "k_sc_list", "k_mt"} <= {k for _, k, _ in found}
    bad = [(f, k, v) for f, k, args in found for v in re.findall(r"__restrict__\s+(\w+)", args)
           if (k, v) not in FINISHED]
    assert not bad


def test_helpers_of_the_adjoint_steps():
    text = (CSRC / "adjoint.cu").read_text()
    args = re.search(r"void gather\(([^)]*)\)", text).group(1)
    assert "__restrict__" not in args
