"""Registers of the built kernels, from the compiler's report that the build
keeps beside each object: kernels that every small product goes through hold
their state in registers. (A shared helper that kept more loads in flight once
made the request loop spill 452 bytes and the reduction kernels run up to 1.5
times longer.)
"""
import os
import re

import pytest

import tapp_b200


def spill_bytes(source):
    """{mangled kernel name: bytes of spill stores} of one CUDA source"""
    path = os.path.join(tapp_b200.PKG_DIR, "build", f"cuda_{source}.ptxas.txt")
    if not os.path.exists(path):
        pytest.skip("no compiler report: the library was not built in this tree")
    with open(path) as f:
        text = f.read()
    return {m[1]: int(m[2]) for m in re.finditer(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores", text, re.S)}


@pytest.mark.parametrize("kernel", ["k_request_loop", "k_elementwise_groupI", "k_reduceIfLb0E", "k_reduceIfLb1E",
                                    "k_reduceIdLb0E"])
def test_shared_element_code_does_not_spill(kernel):
    found = {n: b for n, b in spill_bytes("generic").items() if kernel in n}
    assert found and not any(found.values()), found
