"""Kernels that may start while the kernel before them is still writing (programmatic dependent launch): what that kernel
writes is read with ordinary loads.  ``__ldg`` (ld.global.nc) is defined only for data that is read-only for the
reading kernel's whole lifetime, which those buffers are not; no run on a device can show the difference."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ascend_kernel_b200", "csrc")


def _text(name):
    return open(os.path.join(CSRC, name)).read()


def test_row_sums_are_read_with_ordinary_loads():
    text = _text("grouped_gemm.cu")
    assert "launch_dependent(grouped_gemm_kernel" in text
    reads = re.findall(r"(\w+)\(a\.rowsum", text)
    assert reads and set(reads) == {"__ldca"}


def test_prepared_x_is_read_with_ordinary_loads():
    """x as scaled f16 and the rows' exponents, written by the fp4 prepass (PATH 1 is the kernel launched behind it)."""
    text = _text("grouped_gemv.cu")
    assert "launch_dependent(grouped_gemv_kernel<MODE, PATH>" in text
    loads = re.findall(r"const uint4 v = (.*?\(src \+ i\).*);", text)
    assert loads == ["PATH == 1 ? __ldca(src + i) : __ldg(src + i)"]
    assert not re.search(r"__ldg\(a\.xexp", text)
