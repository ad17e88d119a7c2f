"""bench.py's reference arm where the reference's libraries are not built: one line that says so, and exit code 0."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import sys
sys.argv = ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"]
sys.path.insert(0, %r)
from oracle import ref
ref.REF_DIR = %r
import bench
bench.main()
"""


def _run(tmp_path, env):
    return subprocess.run([sys.executable, "-c", RUN % (ROOT, str(tmp_path))], cwd=ROOT, env=dict(os.environ, **env),
                          capture_output=True, text=True, timeout=600)


def test_reference_arm_without_its_libraries(tmp_path):
    r = _run(tmp_path, {})
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout)
    assert d["impl"] == "reference" and set(d) == {"impl", "unavailable"}
    assert "libref_" in d["unavailable"] and "\n" not in d["unavailable"]


def test_other_ranks_stay_silent_without_the_libraries(tmp_path):
    r = _run(tmp_path, {"RANK": "1", "WORLD_SIZE": "2"})
    assert r.returncode == 0 and r.stdout.strip() == "", r.stderr[-2000:]
