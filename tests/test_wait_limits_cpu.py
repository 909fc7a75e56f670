"""The limit of the waits inside kernels (WaitLimits): a block whose wait gave up
waits under the same limit for its copies in flight before its shared and tensor
memory are released, so however short a caller makes the limit, the kernels get
one that such copies (microseconds) meet."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = r"""
#include "kernels.cuh"
#include <cstdio>
int main() {
  for (unsigned long long ns : {0ull, 1ull, 99999ull, 100000ull, 2000000ull, 1ull << 40}) {
    dnspir::WaitLimits l;
    l.wait_ns = ns;
    printf("%llu\n", (unsigned long long)l.ns());
  }
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_kernels_get_at_least_a_tenth_of_a_millisecond(tmp_path):
    src, exe = tmp_path / "limits.cu", tmp_path / "limits"
    src.write_text(SOURCE)
    subprocess.check_call([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "dnspir_b200", "csrc"),
                           "-o", str(exe), str(src)])
    got = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split()]
    assert got == [2_000_000_000, 100_000, 100_000, 100_000, 2_000_000, 1 << 40]
