"""Rules that the native sources keep and that no run on one device and one thread would show."""
import os
import re

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "square-wheel_gb300")
SOURCES = sorted(os.path.join(d, f) for d in ("csrc", "host") for f in os.listdir(os.path.join(PKG, d)) if f.endswith((".cu", ".cuh", ".cpp", ".h")))


def _code(path):
    """The file without comments, line numbers kept."""
    text = open(os.path.join(PKG, path)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)


@pytest.mark.parametrize("path", SOURCES)
def test_no_plain_static_variable_in_a_function(path):
    """What a function remembers between calls holds for one device and races between threads: it belongs to the object
    it is about, or is constant, or atomic and kept by device."""
    bad = [(i + 1, line.strip()) for i, line in enumerate(_code(path).split("\n"))
           if re.match(r"[\t ]+static (?!const|std::atomic|__device__|_assert)", line) and "(" not in line.split("=")[0].split("{")[0]]
    assert not bad, bad
