"""Kernels launched ahead of their predecessor's end (grid_dep_wait) must reach its output through plain pointers: behind
const __restrict__ or __ldg a load may take the non-coherent path, and a __restrict__ pointer's loads may be moved above
the wait.  Checked in the sources: such a kernel may qualify only arrays that were complete before its predecessor started,
and outputs that it does not read."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chapsim2_b200", "csrc")
# tables written when the handle is made; an output
QUALIFIED = {"ysolve_kernel": {"Zr", "D", "pa"}, "ysolve_lines_kernel": {"Zr", "D", "pa"},
             "spectral_divide_kernel": {"k2x", "k2y", "k2z"}, "irfft_rows_kernel": {"out"}, "cfft_lines_kernel": set(),
             "fz_project_kernel": set()}


def _kernels():
    """(name, parameter list, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", src):
            i = m.end()
            sig = re.compile(r"\s*void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\s*\(").match(src, i)
            if not sig:
                continue
            depth, j = 1, sig.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(src[j], 0)
                j += 1
            params = src[sig.end():j - 1]
            body = src.index("{", j)
            depth, k = 1, body + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[k], 0)
                k += 1
            yield sig.group(1), params, src[body:k]


def test_predecessor_data_is_unqualified():
    seen = set()
    for name, params, body in _kernels():
        if "grid_dep_wait()" not in body:
            continue
        seen.add(name)
        allowed = QUALIFIED[name]
        restricted = set(re.findall(r"__restrict__\s*(\w+)", params + body))
        assert restricted <= allowed, (name, restricted - allowed)
        ldg = {re.match(r"[\s(&*]*(\w+)", a).group(1) for a in re.findall(r"__ldg\(([^;]*)", body)}
        assert ldg <= allowed, (name, ldg - allowed)
    assert seen == set(QUALIFIED)
