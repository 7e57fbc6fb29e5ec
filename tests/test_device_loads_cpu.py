"""The step kernel is launched while the kernel before it may still run, so what
that kernel writes - the state, inlet planes, the tau correction - is never read
with read-only loads, whose data no running kernel may write.  The solid masks,
complete before the call that sets them returns, may be (bit_at)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "entropicthreadsafe_b200", "csrc")


@pytest.mark.parametrize("name", ("tslb_device.cuh", "tslb_step.cuh"))
def test_read_only_loads_are_of_the_masks(name):
    text = open(os.path.join(CSRC, name)).read()
    body = re.search(r"bool bit_at\(.*?\n}\n", text, re.S)
    if body:
        text = text.replace(body.group(0), "")
    code = "\n".join(line.split("//")[0] for line in text.split("\n"))
    assert not re.findall(r"__ldg|ld\.global\.nc|__ldcv", code)
