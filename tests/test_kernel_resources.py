"""What kernels that count on several CTAs a multiprocessor are compiled to."""

from __future__ import annotations

import re
import subprocess

import pytest

from litinfer_b200.csrc import build

REGISTERS, THREADS = 65536, 192


def compiled(source):
    """Mangled name of every kernel of a source -> (registers, bytes of spill stores)."""
    try:
        nvcc = build.find_nvcc()
    except build.BuildError:
        pytest.skip("no nvcc")
    cmd = [nvcc, *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", str(build.CSRC), "-c", str(build.CSRC / source), "-o", "/dev/null"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out, name, spilled = {}, None, 0
    for line in (r.stdout + r.stderr).splitlines():
        if m := re.search(r"Compiling entry function '(\w+)'", line):
            name = m.group(1)
        elif m := re.search(r"(\d+) bytes spill stores", line):
            spilled = int(m.group(1))
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            out[name] = (int(m.group(1)), spilled)
    return out


def test_two_ctas_of_the_split_streaming_product_fit_a_multiprocessor():
    """17 to 64 tokens, k split over clusters: with one CTA a multiprocessor the clusters of many shapes do not run all at once."""
    found = 0
    for name, (registers, spilled) in compiled("gemv_tcgen05.cu").items():
        m = re.search(r"gemv_tcgen05_kernelILi(\d+)E.+?Li(\d)ELb1E", name)              # tokens a tile, epilogue, split
        if not m or int(m.group(1)) < 32:
            continue
        found += 1
        granted = -(-registers // 8) * 8 * THREADS
        assert 2 * granted <= REGISTERS, f"{name}: {registers} registers"
        if m.group(2) == "2":                                                           # the sum into the residual stream
            assert spilled == 0, f"{name}: {spilled} bytes spilled"
    assert found >= 14
