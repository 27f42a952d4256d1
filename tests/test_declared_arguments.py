"""The types that the Python side declares for the library's functions are those of their prototypes (no GPU, no library)."""
import os
import re

import pytest

from hymt2sharp_b200.kernels import build, ops


@pytest.mark.parametrize("name", sorted(ops._DECLARED))
def test_declared_types_are_the_prototypes(name):
    source = "".join(open(os.path.join(build.CSRC, f)).read() for f in build.sources())
    found = re.search(r"HYMT2_API int " + name + r"\((.*?)\)\s*\{", source, re.S)
    assert found, f"{name} is not in the sources"
    kind = lambda a: "p" if "*" in a or "cudaStream_t" in a else {"long": "l", "float": "f", "int": "i"}[a.split()[0]]
    assert "".join(kind(a.strip()) for a in found.group(1).replace("\n", " ").split(",")) == ops._DECLARED[name]
