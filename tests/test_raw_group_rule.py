"""How many chunks of a compressed raw frame a warp takes (raw.cu map_group,
built here for the host): the first part of a warp's work is a chain over its
chunks, so small frames spread over more warps, and no frame leaves the device
under 24 warps an SM where it has the chunks for them."""
import ctypes
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    with open(os.path.join(ROOT, "imagestackalignator_b200", "csrc", "raw.cu")) as f:
        text = f.read()
    most = re.search(r"constexpr int MAP_G = \d+;", text)
    body = re.search(r"^int map_group\(.*?\}$", text, re.M | re.S)
    assert most and body, "the rule is not in raw.cu"
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text("#include <algorithm>\n" + most.group(0) + '\nextern "C" ' + body.group(0) + "\n")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "rule.so")).map_group
    fn.argtypes, fn.restype = (ctypes.c_longlong, ctypes.c_int), ctypes.c_int
    return fn


@pytest.mark.parametrize("sms", [1, 108, 148])
def test_chunks_per_warp(rule, sms):
    last = 1
    for n in list(range(0, 40000, 7)) + [10 ** 6, 10 ** 8]:
        g = rule(n, sms)
        assert 1 <= g <= 8 and g >= last  # a warp's lists hold eight chunks
        assert -(-n // g) >= min(n, 24 * sms)
        last = g
    assert last == 8
