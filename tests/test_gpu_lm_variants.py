"""The fused motion statistics (widths up to 128 points, up to 512 samples a shot) against the forward
kernel writing seven K regions followed by the statistics kernel (ME_LM_TWO_PASS=1): bit-identical,
with one and with two samples a thread, and by different kernels (the two-kernel path launches one
more).  Above 128 points both arms take the two kernels.  Each arm runs in a process of its own."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys, json, numpy as np, torch
sys.path.insert(0, sys.argv[1])
from motionest import _lib
from motionest.problem import SenseProblem
from motionest.utils import compute_transform_grids_voxel
lib = _lib.load()
stats, launches = [], []
for (X, Y, Z), n in json.loads(sys.argv[3]):
    C, S = 2, 3
    rng = np.random.default_rng(X * Y + n)
    planes = np.zeros((S, X * Y), bool)
    for s in range(S):
        planes[s, rng.choice(X * Y, n, replace=False)] = True
    def rnd(*sh):
        v = rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
        return torch.as_tensor(v.astype(np.complex64)).cuda()
    kg, rk = compute_transform_grids_voxel((X, Y, Z), [1, 1, 1])
    t = torch.as_tensor(rng.uniform(-0.05, 0.05, (S, 6))).cuda()
    pb = SenseProblem(rnd(C, X, Y, Z), rnd(C, X, Y, Z), planes.reshape(S, X, Y), kg, rk, t)
    x = rnd(Z, X, Y)
    a = lib.me_launch_count()
    stats.append(pb.lm_stats(x, 0).cpu().numpy().ravel())
    launches.append(lib.me_launch_count() - a)
np.save(sys.argv[2], np.concatenate(stats))
print(json.dumps(launches))
"""

# one sample a thread, two, the edges between, lines of each parity of R1, and a width above 128
CASES = [((20, 16, 6), 100), ((33, 24, 5), 256), ((40, 48, 6), 257), ((35, 56, 5), 512),
         ((64, 64, 4), 300), ((30, 88, 5), 400), ((40, 112, 6), 511), ((50, 128, 5), 450),
         ((40, 224, 5), 448)]


def _run(tmp_path, name, env):
    out = tmp_path / f"{name}.npy"
    r = subprocess.run([sys.executable, "-c", _CHILD, str(ROOT), str(out), json.dumps(CASES)],
                       env=dict(os.environ, **env), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return np.load(out).reshape(len(CASES), -1), json.loads(r.stdout.strip().splitlines()[-1])


def test_fused_statistics_equal_two_kernels(tmp_path):
    a, na = _run(tmp_path, "fused", {})
    b, nb = _run(tmp_path, "two", {"ME_LM_TWO_PASS": "1"})
    for case, x, y, k, m in zip(CASES, a, b, na, nb):
        assert m - k == (1 if case[0][1] <= 128 else 0), f"{case}: {k} and {m} launches"
        assert np.array_equal(x, y), f"{case}: {np.abs(x - y).max()}"
