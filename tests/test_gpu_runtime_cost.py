"""What the run-time line passes cost beside the Stockham kernels that they replace: one partial
derivative (12 passes, three with two inputs or outputs) is faster, and the process holds no more
device memory.  Each side runs in a process of its own (ME_GENERIC_FFT is read once per
process); the outputs agree to rounding."""
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
from motionest.transform import RigidTransformDerivativeCuda
from motionest.utils import compute_transform_grids_voxel
torch.zeros(1, device="cuda")
free = torch.cuda.mem_get_info()[0]
p = np.array([0.7, -1.1, 0.4, 0.06, -0.05, 0.08])
us, outs = [], []
for sh, q in json.loads(sys.argv[3]):
    kg, rk = compute_transform_grids_voxel(sh, [1, 1, 1])
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(sh, dtype=torch.complex64, device="cuda", generator=g)
    D = RigidTransformDerivativeCuda(sh, p, kg, rk)
    outs.append(D.apply(x, q).cpu().numpy().ravel())
    t = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            D.apply(x, q)
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 200)
    us.append(sorted(t)[4])
    del D, x
torch.cuda.empty_cache()
np.save(sys.argv[2], np.concatenate(outs))
print(json.dumps({"us": us, "held": free - torch.cuda.mem_get_info()[0]}))
"""

# R2 above 16 along each axis, and a small volume of small radices
CASES = [((27, 125, 216), 0), ((216, 27, 125), 3), ((250, 40, 36), 4), ((36, 40, 250), 5),
         ((40, 50, 36), 4)]


def _run(tmp_path, name, env):
    out = tmp_path / f"{name}.npy"
    r = subprocess.run([sys.executable, "-c", _CHILD, str(ROOT), str(out), json.dumps(CASES)],
                       env=dict(os.environ, **env), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1]), np.load(out)


def test_partials_beside_stockham(tmp_path):
    a, x = _run(tmp_path, "runtime", {})
    b, y = _run(tmp_path, "stockham", {"ME_GENERIC_FFT": "1"})
    # two results within 2e-6 of the same value (the parity tests' bound) are within 4e-6
    assert np.linalg.norm(x - y) < 4e-6 * np.linalg.norm(y)
    for (sh, q), u, v in zip(CASES, a["us"], b["us"]):
        assert u < v, f"partial {q} of {sh}: {u:.0f} us, Stockham {v:.0f} us"
    # modules, plans and the grids' planes; a stack frame of 1 KB alone would take 300 MB
    assert a["held"] < b["held"] + (256 << 20), f"{a['held'] >> 20} MB held"
