"""The place of a spike-history entry (hist_index of csrc/bg3_stdp.cuh), compiled for the host: inside
the ring for every entry the STDP walks ask for, whatever the ring's length, and the reference's
remainder wherever that is not negative (Neurons/AllSpikingNeurons.cpp:182-188)."""
import os
import subprocess

from braingrid_gb300 import build as bgbuild

PROGRAM = r"""
#include <cstdio>
#include "bg3_stdp.cuh"
int main()
{
    long bad = 0, outside = 0;
    for (int ms = 1; ms <= 40; ms++)
        for (int co = 0; co < 6 * ms; co++)
            for (int off = -(ms > 3 ? ms : 3); off <= -1; off++) {
                const int x = bg3::hist_index(co, ms, off), r = (co + ms + off) % ms;
                outside += x < 0 || x >= ms;
                bad += r >= 0 && x != r;
            }
    printf("%ld %ld\n", outside, bad);
}
"""


def test_history_places_stay_inside_the_ring(tmp_path):
    src, exe = str(tmp_path / "places.cu"), str(tmp_path / "places")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.check_call([bgbuild.nvcc()] + bgbuild.ARCH + ["-std=c++17", "-I", bgbuild.CSRC, "-I",
                           os.path.join(bgbuild.ROOT, "include"), src, "-o", exe])
    assert subprocess.check_output([exe]).split() == [b"0", b"0"]
