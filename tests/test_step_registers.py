"""What ptxas says of the fused sweeps (a step's sweep with the next step's neurons in its epilogue)."""
import os
import re

from braingrid_gb300 import build as bgbuild


def test_fused_sweeps_spill_nothing():
    bgbuild.build()
    with open(os.path.join(bgbuild.BUILD, "bg3_step.o.ptxas.txt")) as f:
        text = f.read()
    seen = 0
    for name, spill in re.findall(r"Function properties for (\S+)\n[^\n]*?(\d+) bytes spill stores", text):
        if re.search(r"7k_sweepILi[0-3]ELb1ELi[468]ELi32E", name):
            seen += 1
            assert int(spill) == 0, name
    assert seen >= 3
