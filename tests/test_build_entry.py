"""build() where the reference tree's place holds an empty directory: the pins
are skipped, as without one."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_with_empty_reference_directory(tmp_path):
    out = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.build()"], cwd=ROOT,
                         env=dict(os.environ, GPB_REFERENCE_TREE=str(tmp_path)), capture_output=True, text=True,
                         timeout=900)
    assert out.returncode == 0, out.stderr
