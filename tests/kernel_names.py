"""Kernel families that a step of a run launches (spm_profile_kernels)."""
import ctypes as C
import json

from kapsel3_b200 import _native as N


def step_kernels(run):
    """Takes one step with profiled direct launches; the set of their names."""
    buf = C.create_string_buffer(1 << 16)
    N.check(run.L.spm_profile_kernels(run.h, 1, buf, len(buf)), "spm_profile_kernels")
    return {k["name"] for k in json.loads(buf.value)["kernels"]}
