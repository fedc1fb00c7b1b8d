"""What the build counts as a source file's inputs: a change of a header has to
recompile every file that includes it, or objects with different layouts of a
struct would be linked together."""
import importlib
import os
import re

import conftest
import pytest

build = importlib.import_module(conftest.PKG_NAME + ".build")
SOURCES = build.LIB_SOURCES + build.CLI_SOURCES


def _included(path, seen):
    """The project headers that the compiler reads for a file (quoted includes, beside it or in the public folder)."""
    for name in re.findall(r'#include "([^"]+)"', open(path).read()):
        for folder in (os.path.dirname(path), build.INCLUDE):
            p = os.path.normpath(os.path.join(folder, name))
            if os.path.exists(p):
                if p not in seen:
                    seen.add(p)
                    _included(p, seen)
                break
    return seen


@pytest.mark.parametrize("src", SOURCES)
def test_every_header_is_an_input(src):
    path = os.path.normpath(os.path.join(build.CSRC, src))
    seen = set()
    build._newest_input(path, seen)
    assert _included(path, set()) | {path} <= seen


def test_public_header_is_an_input_of_the_programs():
    header = os.path.normpath(os.path.join(build.INCLUDE, "rihvr.h"))
    for src in build.CLI_SOURCES:
        seen = set()
        build._newest_input(os.path.join(build.CSRC, src), seen)
        assert header in seen, src
