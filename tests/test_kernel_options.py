"""Compile-time options of the kernels are values with a default.  A branch of the preprocessor that the default leaves out is
never built, and no longer builds after a while."""
import os
import re

from test_kernel_ordering import CSRC


def test_no_branch_that_is_never_built():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            lines = [line.strip() for line in f]
        at = [(i, line) for i, line in enumerate(lines) if re.match(r"#\s*(if|else|elif|endif)", line)]
        while at:
            (i, head), (j, tail) = at[:2]
            guard = re.fullmatch(r"#ifndef (MXDSA_\w+)", head)
            assert guard and tail == "#endif" and j == i + 2 and re.match(r"#define " + guard[1] + r"\b", lines[i + 1]), (name, i + 1, head)
            at = at[2:]
