"""Kernel attributes are set once on every device of a process, not once per
process (no GPU: the rule runs on made-up device ordinals), and no kernel that
opts in to more shared memory goes around it."""
import ctypes
import os
import re

from electrodrive_gb300 import build


def test_once_per_device_rule(edlib):
    res = (ctypes.c_int64 * 3)()
    assert edlib.edfmm_device_once_selfcheck(res) == 0
    assert list(res) == [1, 1, 1]


def test_every_shared_memory_opt_in_is_per_device():
    uses = []
    for name in sorted(os.listdir(build.CSRC)):
        with open(os.path.join(build.CSRC, name)) as f:
            uses += [name] * len(re.findall(r"cudaFuncSetAttribute\s*\(", f.read()))
    assert uses == ["edfmm_internal.cuh"]  # allow_smem
