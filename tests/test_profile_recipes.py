"""The profiler commands recorded under profiles/: every one leaves the clocks alone, and one that
collects more than the launches' durations captures one kernel and at most three launches."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FILES = sorted(glob.glob(os.path.join(ROOT, "profiles", "*.md")))


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(p) for p in FILES])
def test_captures_are_small(path):
    text = re.sub(r"\\\n\s*", " ", open(path).read())   # continued lines
    # also options quoted in running text, where a command is described instead of listed
    cmds = re.findall(r"^.*\bncu --(?:metrics|set|section).*$", text, re.M)
    cmds += re.findall(r"`--(?:metrics|set|section)[^`]*`", re.sub(r"\n", " ", text))
    assert cmds or "ncu" not in text
    for c in cmds:
        if c.startswith("`"):
            c = c + " --clock-control none"
        assert "--clock-control none" in c, c
        metrics = re.search(r"--metrics (\S+)", c)
        if metrics and metrics.group(1).strip("`") == "gpu__time_duration.sum" and "--set" not in c and "--section" not in c:
            continue
        count = re.search(r"\s-c (\d+)", c)
        assert count and int(count.group(1)) <= 3 and re.search(r"\s-k ", c), c
