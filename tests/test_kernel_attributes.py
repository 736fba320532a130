"""A kernel's shared-memory limit (cudaFuncSetAttribute) belongs to one device.

Set behind a flag of the process it is missing on every device but the first,
where the launches are then refused.  It takes two devices to see that happen,
so this reads the sources: no such flag may be there.
"""
import re

import pytest

from ecsprt_gb300 import build as b


@pytest.mark.parametrize("src", sorted(b.CSRC.glob("*.cu")), ids=lambda s: s.name)
def test_no_flag_of_the_process_guards_an_attribute(src):
    text = src.read_text()
    if "cudaFuncSetAttribute" not in text:
        pytest.skip("sets no kernel attribute")
    assert not re.findall(r"static\s+(?:std::atomic<bool>|std::once_flag|bool)\s+\w+\s*[;=[{]", text)
