"""Rules for kernels that may be resident while the kernel in front of them still stores (programmatic dependent
launch), read off the sources."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "tensorlogic_b200", "csrc")
WEIGHTS = {"w", "table"}  # written once, before the call that creates them returns


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = open(path).read()
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", text)


def _kernels(text):
    """(name, parameters, body) of every __global__ function with a body."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\s*\(", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params = text[m.end():at - 1]
        start = at = text.index("{", at) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), params, text[start:at]


def test_dependent_kernels_read_their_operands_through_plain_loads():
    """`const T *__restrict__` and __ldg ask for the read-only path, which is defined for data that nothing writes
    during the kernel's whole life -- the time before its dependency wait included.  Only weights are that."""
    seen = set()
    for path, text in _sources():
        for name, params, body in _kernels(text):
            if not re.search(r"griddepcontrol\.wait|tlc_pdl_\w+\(|pdl_wait\(", body):
                continue
            seen.add(name)
            for p in params.split(","):
                m = re.search(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", p)
                assert not m or (m.group(1) in WEIGHTS and name in ("linear_f16_kernel", "linear_q6k_long_kernel", "embed_kernel")), (path, name, p)
        for line in text.splitlines():  # (the GEMMs' producers and the one-row f16 linear: weight tiles and rows)
            if "__ldg(" in line:
                assert re.search(r"__ldg\((?:reinterpret_cast<const \w+ \*>\()?(?:tile|wr) \+", line), (path, line)
    assert {"gemv_mma_kernel", "frag_rows_kernel", "rms_norm_kernel", "elementwise_kernel", "embed_kernel"} <= seen
