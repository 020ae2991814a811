"""What the kernels' sources must hold whatever the data, checked by reading them: no run shows it, since
it matters only where a barrier is lost."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megcc_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


# Every wait on a barrier is bounded; the outcome of one that ran out must be looked at before
# the next wait's takes its place.
@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_the_outcome_of_a_bounded_wait_is_looked_at(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    forgotten = []
    for wait in re.finditer(r"\bok\s*=[^;{}]*\bmbar_wait\w*\([^;]*;", text):
        after = re.search(r"\bok\b(\s*=(?!=)\s*([^;]*);)?", text[wait.end():])
        if after and after.group(1) and not re.search(r"\bok\b", after.group(2)):
            forgotten.append(text[:wait.start()].count("\n") + 1)
    assert not forgotten, f"{os.path.basename(path)}: waits at lines {forgotten}"


# An int8 ConvBias may have as many pixels as an int counts: rounding them up to tiles must not pass that.
# (fp32: 2^30 at most.)
@pytest.mark.parametrize("path", [p for p in SOURCES if "f32" not in os.path.basename(p)], ids=os.path.basename)
def test_pixels_are_rounded_up_without_overflow(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert not re.search(r"(?<!\(long long\))\ba\.m \+ ", text)
