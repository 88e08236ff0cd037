"""Kernels that may be set up while the kernel before them ends (launch() in csrc/sg_common.cuh)
keep every load behind their wait: each ties its addresses to the value that only the wait
produces, through its block number or through all of its read-only pointer parameters.  A
kernel that drops the value leaves that to the compiler's handling of asm clobbers."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "splinegrids.jl_gb300", "csrc")


def _sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(f) as fh:
            out[os.path.basename(f)] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def _kernels(sources):
    """name -> (parameters, body) of every __global__ function."""
    found = {}
    for text in sources.values():
        for m in re.finditer(r"__global__[^;{}]*?\b(k_\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            j = text.index("{", i)
            depth, e = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[e], 0)
                e += 1
            found[m.group(1)] = (params, text[j:e])
    return found


def test_every_overlapped_kernel_ties_its_loads_to_the_wait():
    sources = _sources()
    kernels = _kernels(sources)
    text = "\n".join(sources.values())
    launched = set(re.findall(r"\blaunch\(\s*(k_\w+)", text)) | \
        set(re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(k_\w+)", text))
    assert len(launched) >= 20 and launched <= set(kernels)
    bad = []
    for name in sorted(launched):
        params, body = kernels[name]
        if re.search(r"(\+|\+=)\s*grid_start\(\)", body):  # the block number
            continue
        var = re.search(r"\b(\w+) = grid_start\(\);", body)  # a variable that is added to what they follow from
        if var and re.search(r"\+= " + var.group(1) + r"\b", body[var.end():]):
            continue
        args = re.findall(r"\bgrid_start\(([^()]*)\)", body)
        passed = {a.strip() for a in args[0].split(",")} if len(args) == 1 else set()
        read_only = set(re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
        if not passed - {""} or not read_only <= passed:
            bad.append(name)
    assert not bad, f"kernels whose loads are not tied to the wait: {bad}"
