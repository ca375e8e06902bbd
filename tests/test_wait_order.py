"""Every kernel that may start before the one ahead of it has finished reads that kernel's results only behind its wait.

``griddepcontrol.wait`` alone does not hold the compiler to that: a load through a ``const __restrict__`` parameter counts
as invariant and may be moved above it.  ``after_wait`` names the pointers that are re-materialised behind the wait; this
reads the sources and asks that no such parameter of a waiting kernel is missing from it.  Exempt are parameters that are
read by volatile asm alone (``ldg_nc``, bulk copies), which keeps its place behind the wait, and those whose addresses
are computed from values that were read behind it."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tensorfold_b200" / "csrc"
FILES = ["exl3.cu", "experts_decode.cu", "experts_prefill.cu", "pack.cu", "peer.cu", "routing.cu"]
VOLATILE_READS = {"router_kernel": {"W"}, "router_rows_kernel": {"W"}, "router_mma_kernel": {"W"}, "route_kernel": {"W"},
                  "decode_kernel": {"W"}, "prefill_kernel": {"W"}}
# read and counted up by one kernel of a step, read by the next
COUNTERS = {"combine_push_kernel": {"step"}, "peer_push_kernel": {"step"}}
# addresses that hang on a value read behind the wait: the input scales of the pair's expert
DEPENDENT_ADDRESSES = {"exl3_prologue_kernel": {"suh0", "suh1"}}


def kernels(text: str) -> list[tuple[str, str, str]]:
    """(name, parameters, body) of every kernel."""

    text = re.sub(r"//[^\n]*", "", text)
    found = []
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?=[^()]*(?:\([^()]*\)[^()]*)*\)\s*\{)", text):
        if m.group(1) == "__launch_bounds__":
            continue
        close = text.index(")", m.end())
        at = text.index("{", close)
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        found.append((m.group(1), text[m.end():close], text[at:end]))
    return found


def untied(name: str, params: str, body: str) -> set[str]:
    """Parameters whose loads the compiler may move above the kernel's wait."""

    if "pdl_wait()" not in body:
        return set()
    invariant = {p.split()[-1].lstrip("*&") for p in params.split(",") if "__restrict__" in p and "const" in p}
    invariant |= COUNTERS.get(name, set())
    tied = {n.strip() for call in re.findall(r"after_wait\(([^)]*)\)", body) for n in call.split(",")}
    return invariant - tied - VOLATILE_READS.get(name, set()) - DEPENDENT_ADDRESSES.get(name, set())


@pytest.mark.parametrize("file", FILES)
def test_dependent_pointers_are_tied_to_the_wait(file):
    found = kernels((CSRC / file).read_text())
    assert any("pdl_wait()" in body for _, _, body in found)
    missing = {name: sorted(untied(name, params, body)) for name, params, body in found}
    assert not {n: p for n, p in missing.items() if p}
