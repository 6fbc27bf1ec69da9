"""The rules that choose a kernel or its CTAs by the warps that an SM holds, against the registers that the compiler gives the kernels."""
import functools
import os
import re
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@functools.lru_cache(maxsize=None)
def registers(source):
    """Kernel (demangled, without its arguments) -> registers per thread, as ptxas prints them."""
    from binarybrain_b200 import build
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None or shutil.which("c++filt") is None:
        pytest.skip("no nvcc")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xcompiler", "-fPIC")]
    with tempfile.TemporaryDirectory() as out:
        text = subprocess.run([nvcc, *flags, "-Xptxas", "-v", "-cubin", os.path.join(build.CSRC, source), "-o", os.path.join(out, "out.cubin")], check=True,
                              capture_output=True, text=True).stderr
    names = re.findall(r"Compiling entry function '(\w+)'", text)
    plain = subprocess.run(["c++filt"], input="\n".join(names), capture_output=True, text=True, check=True).stdout.split("\n")
    counts = [int(n) for n in re.findall(r"Used (\d+) registers", text)]
    assert len(names) == len(counts) > 0
    return dict(zip(plain, counts))


# (a quarter of an SM's 65536 registers belongs to each of its four schedulers, whose warps take them in units of 8 a thread)
@pytest.mark.parametrize("source,kernel,warps,kernels", [
    ("binary_mode.cu", r"k_small_binary_forward<\w+(, 64)?>", 64, 2), ("binary_mode.cu", r"k_small_binary_forward<\w+, 48>", 48, 1),
    ("binary_mode.cu", r"k_small_binary_backward<\w+, \w+(, 24)?>", 24, 4), ("binary_mode.cu", r"k_small_binary_backward<\w+, \w+, 16>", 16, 2),
    ("lut6_small.cu", r"k_lut6_small_forward<", 20, 3), ("lut6_small.cu", r"k_lut6_small_backward<", 8, 2)])
def test_an_sm_holds_the_warps_that_a_rule_counts_on(source, kernel, warps, kernels):
    found = {k: n for k, n in registers(source).items() if re.search(kernel, k)}
    assert len(found) == kernels
    for name, n in found.items():
        assert 4 * (16384 // (32 * ((n + 7) // 8 * 8))) >= warps, (name, n)
