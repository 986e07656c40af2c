"""Kernels that are resident while the kernel before them still writes (pdl_wait in csrc/ptx_sm100.cuh) read its results by ordinary
loads: ld.global.nc is for memory that nothing writes during the kernel's lifetime."""
import re

import pytest

from vllm_omni_b200.build import CSRC

TEXT = {f.name: re.sub(r"//[^\n]*", "", f.read_text()) for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}


@pytest.mark.parametrize("name", [n for n, t in TEXT.items() if "pdl_wait" in t or "pdl_begin" in t])
def test_no_read_only_loads(name):
    assert "__ldg" not in TEXT[name] and "ld.global.nc" not in TEXT[name]
