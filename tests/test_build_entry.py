"""build() where the reference's folder is there and its sources are not."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_without_reference_sources(cucm_lib, tmp_path):
    r = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.build()"], cwd=ROOT,
                       env=dict(os.environ, CUCM_REFERENCE_DIR=str(tmp_path)), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
