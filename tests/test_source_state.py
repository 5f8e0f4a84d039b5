"""Host code keeps no state of the process: what the driver keeps per device (a
kernel's shared-memory limit, its occupancy) is asked for once per context."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "ultradmrg_gb300", "csrc")


def test_no_function_local_statics():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        for i, line in enumerate(open(path), 1):
            if re.match(r"\s+static\s+(?!const)[\w:<>]+\s+\w+\s*(=|;|\{)", line):
                found.append("%s:%d" % (os.path.basename(path), i))
    assert not found, found
