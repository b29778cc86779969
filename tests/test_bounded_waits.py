"""Every kernel whose waits have a limit tells somebody when one runs out.

No such wait can be made to run out in a test: what it waits for is always on its way.  So the sources are read instead: a file that waits with a limit sets the
caller's error flag, and the launches that can reach such a kernel have the flag among their arguments.
"""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "fasttalk_llm_microservice_b200" / "csrc"
WAITING = sorted(f.name for f in CSRC.glob("*.cu") if re.search(r"mbar_(wait|sleep)_limited\(", f.read_text()))


@pytest.mark.parametrize("name", WAITING)
def test_a_wait_that_runs_out_marks_the_error_flag(name):
    text = (CSRC / name).read_text()
    assert re.search(r"\*(a\.)?err = 1;", text), f"{name} gives up on a wait without a word"


def test_projections_take_the_engines_flag():
    calls = re.findall(r"launch_linear\(([^;]*)\)", (CSRC / "engine.cu").read_text())
    assert len(calls) > 5 and all("h_kernel_err" in c for c in calls)
