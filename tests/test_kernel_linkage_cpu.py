"""Kernels of files that several units compile are static. Each unit has its own
__constant__ parameters and zone table, and only the units of a context's species
count are written for it; of a kernel template that two units instantiate with external
linkage the linker keeps one, which would run with the other unit's copies."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "openstc-dev_b200" / "csrc"


def _includes(f, seen):
    if f in seen:
        return
    seen.add(f)
    for inc in re.findall(r'^#include "([^"]+)"', f.read_text(), re.M):
        g = CSRC / inc
        if g.exists():
            _includes(g, seen)


def _shared():
    """files that more than one unit compiles"""
    units = {}
    for u in sorted(CSRC.glob("*.cu")):
        seen = set()
        _includes(u, seen)
        for f in seen:
            units.setdefault(f, []).append(u.name)
    return sorted(f for f, us in units.items() if len(us) > 1)


def _external_kernels(text):
    """__global__ definitions without static (the declaration may span lines)"""
    text = re.sub(r"//[^\n]*", "", text)
    out = []
    for m in re.finditer(r"__global__", text):
        head = text[:m.start()]
        head = head[max(head.rfind(";"), head.rfind("}"), head.rfind("#")) + 1:]
        if "static" not in head.split():
            out.append(" ".join(text[m.start():m.start() + 90].split()))
    return out


def test_shared_kernels_have_internal_linkage():
    shared = _shared()
    assert {"kernels.cu", "steady.cuh", "flux.cuh"} <= {f.name for f in shared}
    bad = {f.name: _external_kernels(f.read_text()) for f in shared}
    assert not any(bad.values()), {k: v for k, v in bad.items() if v}
