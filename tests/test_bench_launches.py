"""The launch count that bench.py reports against the step loop's graphs as the engine cuts a run."""
import os
import re

import pytest

from conftest import ROOT


@pytest.mark.parametrize("nsteps", [1, 7, 8, 9, 24, 25, 32, 33, 40, 56, 57, 64, 1000, 2048, 2049])
def test_launches_of_a_run(nsteps):
    import bench
    src = open(os.path.join(ROOT, "pygcmc_b200", "csrc", "engine.cu")).read()
    long, short = map(int, re.search(r"kGraphSteps\[2\] = \{(\d+), (\d+)\}", src).groups())
    steps, need = 0, nsteps
    while need > 0:  # launch_steps
        length = long if need > long - short else short
        steps += length
        need -= length
    assert nsteps <= steps < nsteps + short
    assert bench.run_launches(nsteps, 5) == 2 + 5 * steps
