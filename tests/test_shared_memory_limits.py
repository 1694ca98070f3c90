"""A kernel's limit of dynamic shared memory is a property of the whole process: raised to
one context's own size it can be lowered by another thread's smaller context before the
first one launches, which is then refused.  So the limit is set in two helpers only, to a
size that is fixed per kernel (a template argument of it); launches whose size depends on a
context stay within the default 48 KB."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "timstochrigidbodiessim_b200", "csrc")


def test_limits_are_set_in_the_helpers_only():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        lines = open(path).read().split("\n")
        for i, line in enumerate(lines):
            if "cudaFuncSetAttribute(" in line:
                head = [m.group(1) for m in (re.match(r"int (\w+)\(", h) for h in lines[:i]) if m][-1]
                found.append((os.path.basename(path), head))
    assert found == [("fcm_kspace.cu", "xfft_smem_attr"), ("fcm_packed.cuh", "smem_attr_once")]

