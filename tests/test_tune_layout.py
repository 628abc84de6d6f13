"""The launch-shape table's file (BORA_TUNE_FILE, vare_gb300/csrc/tune.cu) carries the layout that its
shapes and size classes belong to: lines of another layout are passed over, on the CPU."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = "from vare_gb300 import build, flip; build.build(); print(flip.tune_table())"


@pytest.mark.parametrize("lines,rows", [
    ("0 0 5 2 0.010000\n1 0 5 3 0.020000\n", "[]"),                     # the bare groups of the first layout
    ("100 0 5 2 0.010000\n300 0 5 2 0.010000\n", "[]"),                 # other layouts
    ("200 0 5 2 0.010000\n1 0 5 3 0.020000\n201 0 6 3 0.020000\n", "[(0, 0, 5, 2, 0.01), (1, 0, 6, 3, 0.02)]"),
    ("-200 0 5 2 0.01\n299 0 5 2 0.01\n200 0 5 9 0.01\n", "[]"),        # no such group or shape
])
def test_layout(tmp_path, lines, rows):
    path = tmp_path / "tune.txt"
    path.write_text(lines)
    out = subprocess.run([sys.executable, "-c", CODE], env=dict(os.environ, BORA_TUNE_FILE=str(path)), cwd=ROOT,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == rows
