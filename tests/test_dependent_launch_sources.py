"""Kernels that may start under their predecessor's tail (csrc/launch.h) read what it writes by ordinary loads: no
read-only qualifier (const __restrict__, __ldg) on anything but what is older than the pass."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diloco_swarm_b200", "csrc")
OLDER = {"gamma", "beta", "wte", "wpe", "ids", "targets", "mask"}


def kernels():
    """(file, name, parameters) of every kernel that waits for its predecessor."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in text.split("__global__")[1:]:
            m = re.match(r"[^{;]*?(\w+_kernel)\s*\(([^{;]*?)\)\s*\{", part, re.S)
            if m and "pdl_wait()" in part:
                yield os.path.basename(path), m.group(1), m.group(2)


def test_parameters():
    seen = []
    for path, name, params in kernels():
        seen.append(name)
        for p in params.split(","):
            if "const" in p and "__restrict__" in p:
                assert p.split()[-1].lstrip("*") in OLDER, (path, name, p.strip())
    for name in ("layernorm_fwd_kernel", "layernorm_bwd_kernel", "attention_bwd_kernel", "gemm_kernel", "gemm_split_kernel",
                 "cross_entropy_kernel", "head_rows_kernel"):
        assert name in seen, seen


def test_device_functions():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        if os.path.basename(path) in ("optim.cu", "collectives.cu"):         # never launched dependently
            continue
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__ldg\(([^;]*)", text):
            assert "bias" in m.group(1), (path, m.group(0)[:80])
        for m in re.finditer(r"__device__ __forceinline__ [^{;]*?\(([^{;]*?)\)\s*\{", text, re.S):
            assert not re.search(r"const [^,]*__restrict__", m.group(1)), (path, m.group(0)[:120])
