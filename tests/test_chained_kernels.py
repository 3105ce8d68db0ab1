"""Kernels that are placed while the kernel before them still runs read its output through plain pointers: const
__restrict__ would let the compiler load it by the path for data that nobody writes while the kernel runs."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "n-queens_gb300", "csrc")
# written by the host before the first kernel of the chain
UPLOADED = {"starts", "qs", "ends"}


def test_no_restrict_on_what_the_kernel_before_writes():
    found = 0
    for name in ("nq_kernels.cu", "nq_gen.cu", "nq_unique.cu"):
        src = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(([^{;]*)\)\s*\{", src):
            body, depth, i = "", 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                body += src[i]
                i += 1
            if "chain_wait()" not in body:
                continue
            found += 1
            named = set(re.findall(r"const [\w<>:]+(?: [\w<>:]+)*\s*\*\s*__restrict__\s+(\w+)", m.group(2) + body))
            assert named <= UPLOADED, (m.group(1), named)
    assert found >= 8
