"""Kernels launched as a chain (launch_chained) may start while the kernel ahead
of them still writes.  A read-only promise (``const ... __restrict__``) on a
buffer that a kernel of the chain writes would let the compiler take the
read-only load path, whose data must not change while the kernel lives: no such
buffer carries it, as a parameter of a chained kernel or in its argument
structs."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "dgswem_b200" / "csrc"
SOURCES = ["adjoint.cu", "hydro_kernels.cuh", "hydro_p2.cuh", "kernel_launch.inc"]
# states, flags, cotangents and node bounds: what stages, limiter and reverse
# sweep hand from kernel to kernel
WRITTEN = {"q", "qin", "qout", "qhist", "rhist", "rout", "wd", "nu", "lam", "lam_j", "mm", "arg", "lb", "nb", "minmax",
           "eb", "ib_rhs", "ef"}
PROMISE = re.compile(r"\bconst\s+\w+\s*\*\s*__restrict__\s+(\w+)")


def _text(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_no_read_only_promise_on_written_buffers():
    text = {s: _text(s) for s in SOURCES}
    chained = set()
    for t in text.values():
        chained |= set(re.findall(r"launch_chained\(\s*(\w+)", t)) - {"void", "k"}
        chained |= set(re.findall(r"auto\* k = [^;]*?\b((?:stage|p2)_\w+)<", t))
    assert {"limit_wetdry", "node_minmax", "stage_p1", "p2_tile", "limit_vjp", "edge_vjp"} <= chained
    bad = []
    for s, t in text.items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)\s*)?(\w+)\(([^{]*)\)\s*\{",
                             t):
            if m.group(1) in chained:
                bad += [(m.group(1), p) for p in PROMISE.findall(m.group(2)) if p in WRITTEN]
    header = _text("hydro_device.cuh")
    for struct in ("StageArgs", "LimitArgs", "P2Args", "AdjArgs", "SspAdjArgs"):
        body = re.search(r"struct %s \{(.*?)\n\};" % struct, header, re.S).group(1)
        bad += [(struct, p) for p in PROMISE.findall(body) if p in WRITTEN]
    assert not bad
