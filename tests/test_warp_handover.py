"""One lane arrives on an mbarrier for its whole warp, to hand over what all 32
lanes wrote or read.  Its arrive orders only what is already ordered before it,
which is what __syncwarp does for the other lanes' accesses and a vote
(__any_sync, __all_sync) does not: the kernels' sources, read for it."""
import glob
import os
import re

import pytest

from conftest import ROOT

# the barriers over which whole warps hand shared or tensor memory to others
HANDED = re.compile(r"mbar_arrive(_rank)?\((smem_u32\(&?(facfull|facempty|ufull|pempty|accempty)\b"
                    r"|uf\b)")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(ROOT, "qld_b200", "csrc",
                                                               "ld_*m*.cu"))
                                        + [os.path.join(ROOT, "qld_b200", "csrc", "ld_batch.cu")]),
                         ids=os.path.basename)
def test_a_warp_syncs_before_one_lane_arrives(path):
    with open(path) as f:
        lines = [line.split("//")[0].strip() for line in f]
    lines = [line for line in lines if line and not line.startswith("#")]
    found = 0
    for at, line in enumerate(lines):
        if not HANDED.search(line):
            continue
        lead = at
        while not lines[lead].startswith("if (lane == 0)"):
            lead -= 1
            assert at - lead < 4, f"{line}: not under `if (lane == 0)`"
        assert lines[lead - 1] == "__syncwarp();", f"{lines[lead - 1]} before {line}"
        found += 1
    assert found >= 2
