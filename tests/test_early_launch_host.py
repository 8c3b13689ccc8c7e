"""Kernels that start beside the end of the kernel before them (previous_done in pr_internal.cuh) read that
kernel's output while it is, for a part of their own run, still being written.  __restrict__ would let
the compiler load it through the non-coherent path or above the wait, with stale values as the
result, so such kernels and what they call may have it on layouts and coefficients alone.
"""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "porerad_b200" / "csrc"
# written before the chain of early kernels begins: the preconditioner's coefficients, and the table of
# a batch of products, whose launch is an ordinary one
CONSTANT = {"diag", "shift", "items"}


def _functions():
    """(file, name, qualifiers and parameters, body) of every device function and kernel."""

    found = []
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", path.read_text())
        for m in re.finditer(r"__(?:global|device)__[^;{}=]*?(\w+)\s*\(([^{};]*)\)\s*(?:const\s*)?\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            found.append((path.name, m.group(1), m.group(0), text[m.end():at]))
    return found


def test_early_kernels_read_the_stream_s_data_through_plain_pointers():
    functions = _functions()
    early = {name for _, name, _, body in functions if re.search(r"\bprevious_done\(\)", body)}
    while True:  # and the kernels that call them, and what these kernels hand their pointers on to
        callers = {name for _, name, _, body in functions
                   if any(re.search(rf"\b{e}\s*(?:<[^>]*>)?\(", body) for e in early)}
        if callers <= early:
            break
        early |= callers
    bodies = " ".join(body for _, name, _, body in functions if name in early)
    early |= {name for _, name, _, _ in functions
              if name.startswith(("spmv_stream", "stream_load")) and re.search(rf"\b{name}\b", bodies)}
    assert {"k_spmv_stream", "spmv_stream_cta", "stream_load_x", "k_stream_rows", "spmv_stream_rows", "k_pcg_apply",
            "k_pcg_update"} <= early
    for path, name, head, _ in functions:
        if name in early:
            marked = set(re.findall(r"__restrict__\s+(\w+)", head))
            assert marked <= CONSTANT, f"{path}: {name} has __restrict__ on {sorted(marked - CONSTANT)}"
