"""gb300_grouped_shape_for over everything its arguments take, empty and largest dimensions included (in a
child process, so that a crash of the query fails the test)."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import blaze_gb300 as G
big = 2 ** 31 - 1
for elem, shapes in ((8, 4), (4, 5)):
    for m in (0, 1, 7, 33, 256, big - 40, big - 1, big, 2 ** 40):
        for n in (0, 1, 9, 64, big, 2 ** 40):
            for k in (0, 1, 100, 2 ** 40):
                s, rows, cols = G.grouped_shape_for(elem, m, n, k)
                assert 0 <= s < shapes and rows > 0 and cols > 0, (elem, m, n, k, s, rows, cols)
# a long thin product takes the tiles that its own proportions fill, however long it is
assert G.grouped_shape_for(8, big, 16, 64) == G.grouped_shape_for(8, 2 ** 20, 16, 64)
assert G.grouped_shape_for(8, 16, big, 64) == G.grouped_shape_for(8, 16, 2 ** 20, 64)
print("ok")
"""


def test_every_size_is_answered():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
