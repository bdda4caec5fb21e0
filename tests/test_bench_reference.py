"""bench.py --impl reference where the reference's CPU SynC can be neither
loaded nor built: one JSON line that says so, exit code 0."""
import json
import os
import shutil
import subprocess
import sys

from conftest import REPO


def test_reference_arm_without_the_reference(tmp_path):
    for f in ("bench.py", "oracle", "egg-sync_b200"):
        src, dst = REPO / f, tmp_path / f
        if src.is_dir():
            shutil.copytree(src, dst, ignore=shutil.ignore_patterns("_ref", "lib", "csrc", "__pycache__"))
        else:
            shutil.copy(src, dst)
    env = dict(os.environ, EGG_REFERENCE_ROOT=str(tmp_path / "absent"))
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"],
                       cwd=tmp_path, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "unavailable" in line
