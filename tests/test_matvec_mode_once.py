"""A matrix-vector call runs in one mode: the process-wide option, which another
thread may change meanwhile, is read once per entry point and handed on, so that
buffers chosen for one mode's kernel never go to another's."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "tensorkyber_b200", "csrc", "tk_api.cu")


def bodies():
    """{function: body} of tk_api.cu's definitions at the start of a line."""
    with open(SRC) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    return {m.group(1): m.group(0) for m in
            re.finditer(r"^(?:static )?[a-z]\w* (\w+)\([^;{}]*\) \{\n.*?^\}", text, re.M | re.S)}


@pytest.mark.parametrize("entry", ["tk_matvec", "tk_matvec_host", "tk_matvec_host_noalloc"])
def test_the_mode_is_read_once(entry):
    found = bodies()

    def reads(name):
        called = [f for f in found if f != name and re.search(rf"\b{f}\(", found[name])]
        return found[name].count("g_matvec_mode") + sum(reads(f) for f in called)
    assert reads(entry) == 1
