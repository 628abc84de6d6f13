"""The launch-shape table's file (BORA_TUNE_FILE, vare_gb300/csrc/tune.cu) carries the layout that its
shapes and size classes belong to. Lines with the bare group are listed as a first guess and measured
again on live launches; lines of another layout are passed over."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIST = "from vare_gb300 import build, flip; build.build(); print(flip.tune_table())"
STEP = """
from vare_gb300 import flip, scenes
sc = scenes.small(32)
sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_MIXED)
for _ in range(4):
    sim.step(sc.dt)
"""


def _run(code, path):
    out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, BORA_TUNE_FILE=str(path)), cwd=ROOT,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    return out.stdout.strip()


@pytest.mark.parametrize("lines,rows", [
    ("100 0 5 2 0.010000\n300 0 5 2 0.010000\n", "[]"),                 # other layouts
    ("200 0 5 2 0.010000\n1 0 5 3 0.020000\n201 0 6 3 0.020000\n", "[(0, 0, 5, 2, 0.01), (1, 0, 5, 3, 0.02), (1, 0, 6, 3, 0.02)]"),
    ("-200 0 5 2 0.01\n299 0 5 2 0.01\n200 0 5 9 0.01\n-1 0 5 2 0.01\n", "[]"),  # no such group or shape
])
def test_layout(tmp_path, lines, rows):
    path = tmp_path / "tune.txt"
    path.write_text(lines)
    assert _run(LIST, path) == rows


@pytest.mark.gpu
def test_bare_lines_are_measured_again(gpu, tmp_path):
    path = tmp_path / "tune.txt"
    _run(STEP, path)
    entries = [l.split() for l in path.read_text().splitlines()]
    assert entries and all(200 <= int(e[0]) < 206 for e in entries)
    # the same classes as bare lines with an impossible time: replaced by a measurement
    path.write_text("".join(f"{int(e[0]) - 200} {e[1]} {e[2]} {e[3]} 1000.0\n" for e in entries))
    _run(STEP, path)
    again = [l.split() for l in path.read_text().splitlines()]
    assert [e[:3] for e in again] == [e[:3] for e in entries] and all(float(e[4]) < 100.0 for e in again)
    # and read back as measured ones: nothing is written anew
    before = path.read_text()
    _run(STEP, path)
    assert path.read_text() == before
