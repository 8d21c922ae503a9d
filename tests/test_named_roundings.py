"""The sums that decide a process pick name every rounding: a sum left to the compiler is contracted by the code
around it, and a change elsewhere in the kernel then moves picks."""
import os
import re

import pytest

HDR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupythia_b200", "csrc", "cp_integrand.cuh")


@pytest.mark.parametrize("name", ["cp_process_shares", "cp_pick_flavours"])
def test_no_sum_is_left_to_the_compiler(name):
    src = re.sub(r"//[^\n]*", "", open(HDR).read())
    body = re.search(r"\b%s\([^)]*\)\s*\{(.*?)\n\}" % name, src, flags=re.S).group(1)
    body = re.sub(r"(\+\+k|111 \+ k|-c\[k\])", "", body)
    assert not re.findall(r"[+-]", body)
