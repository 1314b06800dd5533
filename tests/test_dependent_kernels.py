"""What a kernel that may start while its producer still runs must not promise.

A kernel launched with launch_dependent reads, after pdl_wait, buffers that
another grid was still writing when it started. A __restrict__ parameter says
that the kernel's own accesses are the only ones for its whole run, which lets
the compiler read it through the non-coherent path, or ahead of the wait. So
no kernel that waits may take one, and every dependent launch is of a kernel
that waits.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "hpc-multigpu-matrixmult_gb300" / "csrc"


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def _kernels():
    """{kernel: (parameters, body)} of every __global__ function in csrc."""
    found = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for g in re.finditer(r"__global__\s+void\s+", text):
            at = g.end()
            bounds = re.match(r"__launch_bounds__", text[at:])
            if bounds:
                at = _closing(text, text.index("(", at), "()") + 1
            name = re.match(r"\s*(\w+)\s*\(", text[at:])
            lp = at + name.end() - 1
            rp = _closing(text, lp, "()")
            lb = text.index("{", rp)
            found[name.group(1)] = (text[lp:rp], text[lb:_closing(text, lb, "{}")])
    return found


def _dependent_launches():
    names = set()
    for path in sorted(CSRC.glob("*.cu")):
        for launch in re.finditer(r"launch_dependent\(\w+,\s*(\w+)", path.read_text()):
            # the slice GEMM's instantiations are launched through a local name
            names.add("tc_slice_gemm_kernel" if launch.group(1) == "kern" else launch.group(1))
    return names


def test_dependent_launches_wait():
    kernels, launched = _kernels(), _dependent_launches()
    assert {"tc_slice_gemm_kernel", "crt_kernel", "residue_split_kernel", "scan_cols_merge_kernel"} <= launched
    for name in launched:
        assert "pdl_wait()" in kernels[name][1], name


def test_waiting_kernels_take_no_restrict_pointers():
    waiting = {name: params for name, (params, body) in _kernels().items() if "pdl_wait()" in body}
    assert set(waiting) >= _dependent_launches()
    for name, params in waiting.items():
        assert "__restrict__" not in params, name
