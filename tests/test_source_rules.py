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


def _enclosing_loop(code, at):
    """Text of the innermost braced loop body around an offset, up to it and after it."""
    depth, i = 0, at
    while i > 0:
        i -= 1
        if code[i] == "}":
            depth += 1
        elif code[i] == "{" and depth:
            depth -= 1
        elif code[i] == "{" and re.search(r"\b(for|while) \([^{}]*$", code[max(0, i - 200):i]):
            break
    end, depth = i, 0
    while True:
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        end += 1
        if depth == 0 or end >= len(code):
            return code[i:end]


@pytest.mark.parametrize("path", [p for p in SOURCES if p.startswith("csrc")])
def test_accumulators_are_loaded_by_converged_warps(path):
    """tcgen05.ld is an instruction of the whole warp: no lane may skip ahead to a loop's next load on its own."""
    code = _code(path)
    for m in re.finditer(r"\bcontinue;", code):
        assert "tmem_ld(" not in _enclosing_loop(code, m.start()), f"line {code[:m.start()].count(chr(10)) + 1}"


def _functions(code):
    """Bodies of the device functions and kernels of a file by name (overloads together)."""
    out = {}
    for m in re.finditer(r"__(?:device|global)__[^;{}]*?\{", code):
        name = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)|__align__\([^)]*\)", "", m.group()))
        if not name:
            continue
        end, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            end += 1
        out[name.group(1)] = out.get(name.group(1), "") + code[m.end():end]
    return out


@pytest.mark.parametrize("path", [p for p in SOURCES if p.endswith(".cu")])
def test_kernels_that_start_early_read_with_plain_loads(path):
    """A kernel launched as a programmatic dependent starts while the one before still writes: what it reads is not read-only
    for its whole lifetime, as the loads of __ldg (ld.global.nc) require."""
    code = _code(path)
    functions = {}
    for f in [path] + [p for p in SOURCES if p.endswith(".cuh")]:
        for name, body in _functions(_code(f)).items():
            functions[name] = functions.get(name, "") + body
    todo = re.findall(r"launch_dependent\((\w+)", code)
    todo = [n for n in todo if n in functions]
    seen = set()
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        assert "__ldg(" not in functions[n], n
        todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\(", functions[n])) if c in functions]
    if "launch_dependent(" in code and path != os.path.join("csrc", "sw_device.cuh"):
        assert seen
