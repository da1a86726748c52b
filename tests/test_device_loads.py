"""The read-only load path (__ldg, ld.global.nc) is for memory that no kernel
writes while the reading grid lives.  A grid launched as a programmatic
dependent is resident while the kernel before it still runs, so only tables
that nothing writes after the library is loaded may be read that way."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "atomiverse_b200", "csrc")
CONSTANT = ("kExp2Tab",)  # __device__ const tables


def test_read_only_loads_are_of_constant_tables():
    found = []
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        code = re.sub(r"//.*", "", open(f).read())
        for m in re.finditer(r"__ldg\s*\(\s*(\w+)|ld\.global\.nc", code):
            if m.group(1) not in CONSTANT:
                found.append((os.path.basename(f), m.group(0)))
    assert not found


def test_no_restricted_kernel_parameters():
    # the compiler may turn reads through a const __restrict__ kernel
    # parameter into read-only loads of its own accord
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        code = re.sub(r"//.*", "", open(f).read())
        for m in re.finditer(r"__global__[^{;]*\{", code):
            assert "__restrict__" not in m.group(0), (os.path.basename(f), m.group(0))
