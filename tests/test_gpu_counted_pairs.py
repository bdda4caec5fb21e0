"""The stats build's count of pairs within eps holds tested pairs only: points
counted with a whole 32-point group are not among them."""
import json
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from eggsync import egg_sync, _lib
rng = np.random.default_rng(0)
d = int(sys.argv[2])
X = np.clip(0.5 + 0.05 * rng.standard_normal((20000, d)), 0, 1).astype(np.float32)
egg_sync(X, float(sys.argv[3]), max_iter=2)
out = (C.c_int64 * 32)()
n = _lib.load().egg_update_counters(out, 32)
print(json.dumps(dict(zip(_lib.UPDATE_COUNTERS, [int(v) for v in out[:n]]))))
"""


@pytest.mark.parametrize("d,eps", [(1, 0.1), (2, 0.2), (3, 0.3), (5, 0.4)])
def test_counted_pairs_are_tested_pairs(d, eps):
    env = dict(os.environ, EGGSYNC_LIB=str(REPO / "egg-sync_b200" / "lib" / "libeggsync_stats.so"))
    r = subprocess.run([sys.executable, "-c", CHILD, str(REPO / "egg-sync_b200"), str(d), str(eps)], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    k = json.loads(r.stdout.strip().splitlines()[-1])
    assert k["groups_in"] > 0 and 0 < k["pairs_in"] <= k["pairs"]
