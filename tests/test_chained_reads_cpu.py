"""Kernels that may start while the one before them still writes (chain_wait)
promise the compiler read-only memory for what is laid out once and for nothing
else, and gather the iterate with ordinary loads."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "knappnet_b200" / "csrc"
LAID_OUT_ONCE = {"coords", "sr", "y_ref"}


def chained():
    """(kernel, its parameters) of every kernel that begins with chain_wait."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for k in re.finditer(r"__global__\s+void\b", text):
            head = text[k.end():text.index("{", k.end())]
            head = re.sub(r"__launch_bounds__\(.*?\)\)?\s*\n", "", head, count=1)
            name, params = re.search(r"(\w+)\s*\((.*)\)\s*$", head, re.S).groups()
            body = text[text.index("{", k.end()):]
            if "chain_wait();" in body[:body.index("\n}")]:
                yield name, params


def test_every_chained_kernel_is_seen():
    names = {n for n, _ in chained()}
    assert {"warp_spmv", "slice_spmv", "split_rows", "lz_project", "lz_subtract", "lz_next",
            "pr_exact_change"} <= names
    text = "".join(p.read_text() for p in CSRC.glob("*.cu*"))
    launched = set(re.findall(r"launch_chained\((\w+)", text)) - {"fnp", "void"}
    assert launched <= names


def test_no_read_only_promise_on_what_is_being_written():
    for name, params in chained():
        for q in re.findall(r"const\s+[\w<>: ]+\*\s*__restrict__\s+(\w+)", params):
            assert q in LAID_OUT_ONCE, (name, q)


def test_gathers_of_the_iterate_are_ordinary_loads():
    text = (CSRC / "common.cuh").read_text()
    loads = re.findall(r" ld_keep\w*\(.*?\n}", text, re.S)
    assert len(loads) == 4
    assert not any(".nc" in x for x in loads)
    assert all("asm volatile(" in x for x in loads)  # not moved before chain_wait's
    for path in ("spmv.cuh", "slice.cuh"):
        for body in re.findall(r"chain_wait\(\);(.*?)\n}\n", (CSRC / path).read_text(), re.S):
            assert "__ldg(" not in body
