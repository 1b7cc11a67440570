"""The kernels of a chain (a step kernel that may start while the step before
it still writes the populations) must not take populations through read-only
loads, which CUDA allows only for data that nothing writes during the kernel's
life: no S::ld / S::ld2 (``__ldg``) and no ``const __restrict__`` population
pointer in such a kernel or in any function it calls. Read from the sources,
since a stale value would show only in a rare interleaving."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flowcraft_b200", "csrc")
FILES = ["storage.cuh", "step_common.cuh", "collide2.cuh", "aa.cuh", "lbm_step.cu", "lbm_step_aa.cu"]


def _functions():
    """name -> text of every function, signature and body (overloads joined)."""
    out = {}
    for f in FILES:
        text = open(os.path.join(CSRC, f)).read()
        text = re.sub(r"//[^\n]*|/\*.*?\*/|^#(?:[^\n]*\\\n)*[^\n]*", "", text, flags=re.S | re.M)
        text = re.sub(r"\bnamespace\s*\w*\s*\{", "", text)
        depth = begin = 0
        for k, ch in enumerate(text):
            if ch == "{":
                depth += 1
            elif ch in "};":
                depth -= ch == "}"
                if depth <= 0:
                    depth, piece = 0, text[begin:k + 1]
                    begin = k + 1
                    sig = re.sub(r"__launch_bounds__\([^;{}]*?\)\s(?=\w)", "", piece.split("{")[0])
                    m = re.search(r"(\w+)\((?!.*\bdecltype)", sig)
                    if ch == "}" and m:
                        out[m.group(1)] = out.get(m.group(1), "") + piece
    return out


FUNCS = _functions()
CHAINED = sorted(n for n, t in FUNCS.items() if "__global__" in t and "step_enter()" in t)


def test_chained_kernels_are_found():
    assert {"k_bulk_pairs", "k_bulk_pairs_learned", "k_bulk_pairs_aa", "k_bulk_pairs_aa_learned"} <= set(CHAINED)
    for n in ("pairs_tile", "boundary_entry", "row_end_cell", "bulk_cell", "plane_cell", "load_plane", "load_pop_i"):
        assert n in FUNCS


@pytest.mark.parametrize("kernel", CHAINED)
def test_populations_come_by_ordinary_loads(kernel):
    todo, seen = [kernel], set()
    while todo:
        name = todo.pop()
        if name in seen:
            continue
        seen.add(name)
        text = FUNCS[name]
        assert not re.search(r"\bS::ld2?\(", text), f"{name}: a read-only load of populations"
        assert not re.search(r"S::T\s*\*\s*__restrict__", text), f"{name}: a __restrict__ population pointer"
        todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", text)) if c in FUNCS]
    assert "load_plane" in seen or "aa_boundary_entry" in seen or "aa_boundary_entry_learned" in seen
