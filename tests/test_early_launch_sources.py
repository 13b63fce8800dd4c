"""Kernels that may come onto the device before their predecessor has ended
(their prologue is blk_chain) overlap, in lifetime, a kernel that still writes
the fields and step scalars they read after the wait.  A load through the
read-only path (__ldg, or a pointer that is both const and __restrict__) is
only defined for data that nothing writes during the kernel's lifetime, so
such kernels may use it for the tables of a plan alone.  Checked on the source
text: the kernels' and their bodies' parameter lists, and every load in the
bodies and in the device functions that they call.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cans-fizzy_b200", "csrc")
# written when the plan is made, by kernels and copies that end before any
# kernel that reads them starts
TABLES = {"lam", "a", "b", "c", "piv", "df", "piv0", "df0", "lpr"}
TABLE_LOAD = re.compile(r"^\s*\(?\s*(?:&pl\.tw|(?:%s)\b)" % "|".join(TABLES))
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        s = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", s, flags=re.S))


def _block(s, at):
    """The brace block that opens at or after position `at`."""
    i = s.index("{", at)
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == "{") - (s[j] == "}")
        if depth == 0:
            return s[at : j + 1]
    raise AssertionError("unbalanced braces")


ALL = {f: _source(f) for f in FILES}
TEXT = "\n".join(ALL.values())
STRUCTS = {m.group(1): _block(TEXT, m.start()) for m in re.finditer(r"\bstruct\s+(\w+)\s*\{", TEXT)}
FUNCS = {}
for m in re.finditer(r"__device__[^;{}()]*?\b(\w+)\s*(?:<[^;{}()]*>)?\s*\([^;{}]*\)\s*\{", TEXT):
    FUNCS.setdefault(m.group(1), []).append(_block(TEXT, m.start()))
KERNELS = re.findall(r"(__global__[^;{}]*\{\s*(\w+)(?:<[^;{}()]*>)?::run\(blk_chain\(\))", TEXT)


def _closure(body):
    """`body` and the device functions it calls, directly or not."""
    seen, todo, out = set(), [body], []
    while todo:
        b = todo.pop()
        out.append(b)
        for name in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", b)):
            if name in FUNCS and name not in seen and name != "run":
                seen.add(name)
                todo += FUNCS[name]
    return out


def test_the_kernels_are_found():
    assert len(KERNELS) >= 25
    assert {"MomentumTile", "AcdiTile", "YoungsTile", "ZSolvePart", "BcAll", "StepReduce"} <= {k[1] for k in KERNELS}


@pytest.mark.parametrize("head,struct", KERNELS, ids=[k[1] for k in KERNELS])
def test_only_plan_tables_take_the_read_only_path(head, struct):
    body = STRUCTS[struct]
    lists = [head] + re.findall(r"\brun\((const Blk&.*?)\)\s*\{", body, flags=re.S)
    assert len(lists) == 2
    for text in lists:
        names = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", text)
        assert set(names) <= TABLES, (struct, names)
    for b in _closure(body):
        for arg in re.findall(r"(?:__ldg|\bLD)\(([^;]*)", b):
            assert TABLE_LOAD.match(arg), (struct, arg.split("\n")[0])
        args = re.match(r"[^{]*", b).group(0)
        names = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", args)
        assert set(names) <= TABLES, (struct, names)
