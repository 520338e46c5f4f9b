"""Kernels that are placed while their predecessors run (launch_chained): they wait before they touch
memory, and promise the compiler nothing about memory that the predecessors still write."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "frehg_gb300", "csrc")


def kernels():
    """name -> (parameter list, body) of every kernel defined in the sources"""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            head, _, rest = text[m.end():].partition("{")
            if ";" in head:
                continue  # a declaration
            name = re.search(r"\b(k\w+)\s*\(", head)
            out[name.group(1)] = (head[name.end():], rest[:rest.find("\n}")])
    return out


def launched():
    names = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"launch_chained\s*\(", text):
            arg = text[m.end():m.end() + 200].split(",")[0] if "?" not in text[m.end():m.end() + 80] \
                else text[m.end():m.end() + 200]
            names |= set(re.findall(r"\bk\w*_\w+", arg))
        names |= set(re.findall(r"auto kernel = [^;]*?(k_sor_solve)", text))
    return names


def test_chained_kernels_wait_first():
    defs = kernels()
    names = {n for n in launched() if n in defs}
    assert len(names) >= 25 and {"k32_line_step", "k_sor_solve", "k_prep_ff_split"} <= names
    for n in names:
        body = defs[n][1]
        assert "grid_begin();" in body, n
        before = body[:body.index("grid_begin();")]
        for line in filter(None, (s.strip() for s in before.split(";"))):  # shared declarations only
            assert "__shared__" in line, (n, line)


def test_chained_kernels_promise_nothing():
    for n, (params, body) in kernels().items():
        if "grid_begin();" in body:
            assert "__restrict__" not in params, n
