"""No TMA load of the library writes to another CTA than its own: the same library runs
with one process per GPU, where cluster multicast loads are not used."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "zquatev_gb300", "csrc")


def test_copies_are_not_multicast():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for copy in re.findall(r"cp\.async\.bulk[^;]*;", text):
            found += 1
            assert ".multicast" not in copy, name
    assert found >= 2
