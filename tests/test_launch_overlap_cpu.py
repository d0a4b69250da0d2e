"""HMC_B200_PDL=0 serialises the passes of a sweep: every launch that may overlap the kernel ahead of it takes
that from its Launch, whose flag the host sets by the switch, or is one of the rebuild's chained kernels."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hoomd_rs_b200", "csrc")


def test_no_pass_overlaps_regardless_of_the_switch():
    launches = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                launches += [(name, m.group(0)) for m in re.finditer(r"\bPassLaunch \w+\(.*?\);", f.read(), re.S)]
    assert len(launches) >= 10
    assert [x for x in launches if re.search(r"[(,]\s*true\s*,", x[1])] == []
