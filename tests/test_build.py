"""The build's list of inputs (what makes the library stale)."""

import re

from fastvid_b200 import build


def test_every_source_and_header_is_an_input():
    have = set(build.SOURCES) | set(build.HEADERS)
    assert have == {p.name for p in build.CSRC.iterdir() if p.suffix in (".cu", ".cuh")}
    for name in have:
        included = re.findall(r'#include "([^/"]+)"', (build.CSRC / name).read_text())
        assert set(included) <= have, name
