"""A kernel whose lanes meet in full-warp votes leaves its loop by a vote too:
every comparison of the clock with the watchdog's bound is one (checked in the
source, since lanes that disagree at the bound cannot be had on purpose)."""
import glob
import os
import re

from conftest import ROOT


def test_watchdog_exits_are_warp_votes():
    found = 0
    for path in glob.glob(os.path.join(ROOT, "billardballraytracing3d_b200", "csrc", "*.cu*")):
        for line in open(path):
            if re.search(r"clock64\(\).*>.*watchdog_cycles", line):
                found += 1
                assert re.search(r"__any_sync\(kFull, clock64\(\)", line), (os.path.basename(path), line.strip())
    assert found == 3   # k_advance, k_walk, k_stage1
