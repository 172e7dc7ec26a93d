"""Tuning files of other kernels: their costs and per-tile weights mean something else, so a mode line
without this build's kernels number leaves the default choice in place, the file loading all the same; a
file that this build saved comes back as it was.  Each case in a child process (the state is the
process's)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import blaze_gb300 as G
L, path, head = G.lib(), sys.argv[1], sys.argv[2]
sizes = [(m, n, k) for m in (5, 9, 24, 60, 100, 250) for n in (6, 20, 33, 130) for k in (8, 40, 200)]
shapes = lambda: [G.grouped_shape_for(e, *s) for e in (8, 4) for s in sizes]
default = shapes()
rows = ["gb300-grouped-tune v2"] + ([head] if head else [])
for d in range(2):  # costs that make the smallest shape look best everywhere
    for a in range(6):
        for b in range(6):
            for c in range(3):
                rows.append("%d %d %d %d 0 1e-6 1 1 1 1 0" % (d, a, b, c))
open(path, "w").write("\n".join(rows) + "\n")
assert L.gb300_grouped_tuning_load(path.encode()) == 0
loaded = shapes()
assert L.gb300_grouped_tuning_save((path + "2").encode()) == 0
assert L.gb300_grouped_tuning_load((path + "2").encode()) == 0
assert shapes() == loaded  # a file of this build's own
print("default" if loaded == default else "smallest" if all(s[0] == 0 for s in loaded) else "other")
"""


@pytest.mark.parametrize("head,expect", [
    ("mode 2 2 -1 -1", "default"),            # saved by earlier kernels: measured costs
    ("mode 0 0 8192 8192", "default"),        # ... and a weight of theirs
    ("mode 2 2 -1 -1 kernels 1", "default"),
    ("mode 2 2", "default"),
    ("mode 2 2 -1 -1 kernels 2", "smallest"),  # these kernels' costs
    ("mode 1 1 -1 -1", "smallest"),            # class shapes stay class shapes
    ("", "smallest"),                          # a table without a mode line: its costs
])
def test_costs_of_other_kernels_are_not_used(tmp_path, head, expect):
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "t.txt"), head], cwd=ROOT, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == expect, (r.stdout, r.stderr)
