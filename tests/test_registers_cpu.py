"""The compiler's own report on kernels whose loops were measured without spills: state that does not fit the registers costs them every tile."""
import os
import re

import pytest

from swiftllm_b200 import build


def _report(source):
    """Bytes of spill stores by kernel, from the last compilation of a source."""
    log = os.path.join(build.OBJ, source + ".ptxas.log")
    if not os.path.exists(log) or os.path.getmtime(log) < os.path.getmtime(os.path.join(build.CSRC, source + ".cu")):
        pytest.skip("not compiled here")
    return {name: int(spill) for name, spill in re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores", open(log).read(), re.S)}


def test_paged_attention_does_not_spill():
    spills = {k: v for k, v in _report("paged_attn_tc").items() if "paged_attn_tc_kernel" in k}
    assert len(spills) == 18                                 # two types, groups of 4, 8 and 16, three ways to number the items
    assert not any(spills.values()), spills
