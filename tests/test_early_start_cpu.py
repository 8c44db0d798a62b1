"""Kernels that start under the tail of the launch ahead (programmatic stream serialisation) are there while
their inputs are being written: no non-coherent loads, which are for memory that nobody writes meanwhile."""
import os
import re

import pytest

from cutlass_flash_atten_fp8_b200.build import CSRC


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["fa8_fwd_sm100.cu", "fa8_decode_sm100.cu", "fa8_quant.cu", "ptx_sm100.cuh"])
def test_no_explicit_non_coherent_load(name):
    assert not re.search(r"__ldg\b|ld\.global\.nc", code(name))


def test_quantisation_reads_through_pointers_that_allow_none():
    kernels = dict(re.findall(r"__global__[^(]*\([^)]*\)\s*(\w+)\(([^{]*)\)\s*\{", code("fa8_quant.cu")))
    assert {"segment_kernel", "amax_kernel", "cast_kernel"} <= set(kernels)
    assert not re.search(r"const \w+\* __restrict__", kernels["segment_kernel"])
    assert "const float* amax" in kernels["cast_kernel"]
