"""Kernel settings belong to a device, not to the process: a limit on dynamic shared memory
set once, for the first device that asks, leaves launches on a second one to fail."""
import os
import re

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")


def test_shared_memory_limits_are_set_per_device():
    uses = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            n = len(re.findall(r"\bcudaFuncSetAttribute\s*\(", text))
            if n:
                uses[name] = n
    # the one call of set_on_device, which keeps a bit per device
    assert uses == {"gb2_internal.cuh": 1}, uses
    text = open(os.path.join(CSRC, "gb2_internal.cuh")).read()
    body = text[text.index("cudaError_t set_on_device"):]
    body = body[:body.index("\n}")]
    assert "cudaGetDevice" in body and "cudaFuncSetAttribute" in body


def test_no_launch_ignores_a_failed_setting():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            text = open(os.path.join(CSRC, name)).read()
            for m in re.finditer(r"\b(allow_smem|prefer_l1)\s*\(", text):
                line = text[text.rfind(";", 0, m.start()) + 1:m.start()]
                assert "=" in line or "return" in line or "GB2_CU(" in line, (name, line)
