"""The bounds-checked build on plans that the small grids do not take: x-lines cut
into segments in the test filter, and several planes per thread with planes left
over."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r'''
from dataclasses import replace
from channel_rl_gb300 import cases as C
from channel_rl_gb300.host import Channel

def run(tag, cases):
    ch = Channel(cases)
    for q, c in enumerate(cases):
        ch.upload(*C.initial_fields(c), inst=q)
    ch.step(1)
    for q in range(len(cases)):
        print(f"FLAGS {tag} {q} {ch.status_flags(q)}")
    ch.close()

for shape in ((576, 7, 4), (1024, 8, 6), (512, 9, 4)):
    run("lines", [C.smaller(C.c1_small(), *shape)])
for les in (C.LES_DSM, C.LES_AMD, C.LES_VREMAN, C.LES_SMAG):
    run("batch", [C.wallmodelled(f"b{n}", *s, 2000.0, les=les, seed=n, x_mass_cte=n % 2)
                  for n, s in enumerate(((64, 41, 18), (54, 16, 54), (96, 33, 18), (36, 24, 54)) * 3)])
print("DONE")
'''


def test_long_lines_and_planes_left_over_stay_in_bounds():
    from channel_rl_gb300 import build
    lib = build.build(variant="bounds")
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=dict(os.environ, CHL_LIBRARY=lib), cwd=ROOT, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    flags = [ln.split() for ln in r.stdout.splitlines() if ln.startswith("FLAGS")]
    assert "DONE" in r.stdout and len(flags) == 3 + 4 * 12
    assert not [f for f in flags if int(f[3]) != 0]
