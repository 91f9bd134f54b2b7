"""Which loads of the kernels are non-coherent (``__ldg``), read from their source.

The kernels of a step are launched with programmatic dependent launch: they are resident
while the kernel that writes their state still runs.  ``__ldg`` promises data that is
constant for the kernel's lifetime, and the compiler may move it above the kernel's wait
for its predecessor, so it may name geometry and connectivity only.
"""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "raven.jl_b200", "csrc")

# element geometry, volume and surface metrics, neighbour table, general face map
CONSTANT = ("eg", "vg", "sg", "P.nbr", "A.nbr", "P.vmapP", "A.sgeo")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            yield name, re.sub(r"//[^\n]*", "", f.read())


def test_ldg_reads_only_what_no_kernel_writes():
    found = [(name, m.group(1)) for name, text in _sources() for m in re.finditer(r"__ldg\(\s*([\w.>-]+)", text)]
    assert found
    assert [x for x in found if x[1] not in CONSTANT] == []


def test_no_hand_written_non_coherent_load():
    assert [name for name, text in _sources() if "ld.global.nc" in text] == []
