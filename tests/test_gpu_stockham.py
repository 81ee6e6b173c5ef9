"""The Stockham kernels (line_pass_kernel, sense_fwd_kernel, sense_adj_kernel), which lengths without
any two-stage plan take (245 and some above 256), on every length by ME_GENERIC_FFT=1: rigid
transforms and partials (all pass modes) against the FP64 oracle, the SENSE forward and adjoint
against complex128 at each number of samples a thread (1, 2, 4, 8) and of accumulators a thread (4,
8, 16), and the seven-volume statistics against the default kernels'.

Tolerances: 2e-6 for ten to twelve passes, as in the parity tests of the other engines.  SENSE: the
sums along x take one rounding a row of a running sum (up to 100 rows: 6e-8 sqrt(100 / 2) / 2, about
2e-7) and the FFT along y some ten more: 1e-6 has room.  Statistics: sums of products of two such
values, 1e-5 of the largest."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys, json, numpy as np, torch
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from conftest import rel_l2
from oracle import Oracle, transform_grids
import motionest
from motionest import _lib
from motionest._lib import ptr
from motionest.problem import SenseProblem
from motionest.utils import compute_transform_grids_voxel
O = Oracle(np.complex128)
out = {"transforms": [], "sense": [], "stats": []}
p = np.array([0.7, -1.1, 0.4, 0.06, -0.05, 0.08])
for sh in ((7, 9, 16), (24, 13, 35), (1, 2, 3), (64, 5, 11), (245, 3, 8)):
    rng = np.random.default_rng(sum(sh))
    x = (rng.standard_normal(sh) + 1j * rng.standard_normal(sh)).astype(np.complex64)
    kg, rk = transform_grids(sh, [1, 1, 1])
    T = motionest.RigidTransformCudaOptimzied(p, kg, rk)
    D = motionest.RigidTransformDerivativeCuda(sh, p, kg, rk)
    e = [rel_l2(T.apply(x), O.rigid_apply(x, p, kg, rk)),
         rel_l2(T.adjoint(x), O.rigid_adjoint(x, p, kg, rk))]
    e += [rel_l2(D.apply(x, q), O.rigid_derivative(x, p, q, kg, rk)) for q in (1, 3, 4, 5)]
    out["transforms"].append(e)
for (X, Y), n in (((9, 7), 20), ((32, 32), 256), ((32, 60), 257), ((33, 100), 600), ((100, 45), 1025),
                  ((40, 64), 2048)):
    C, Z, S = 3, 2, 2
    rng = np.random.default_rng(X * Y)
    planes = np.zeros((S, X * Y), bool)
    for s in range(S):
        planes[s, rng.choice(X * Y, n, replace=False)] = True
    g = torch.Generator(device="cuda").manual_seed(X)
    def rnd(*sh):
        return torch.randn(sh, dtype=torch.complex64, device="cuda", generator=g)
    kg, rk = compute_transform_grids_voxel((X, Y, Z), [1, 1, 1])
    t = torch.as_tensor(rng.uniform(-0.05, 0.05, (S, 6))).cuda()
    mps = rnd(C, X, Y, Z)
    pb = SenseProblem(rnd(C, X, Y, Z), mps, planes.reshape(S, X, Y), kg, rk, t)
    U, K = rnd(S, Z, X, Y), torch.empty(S * n * C * Z, dtype=torch.complex64, device="cuda")
    W, V, st = torch.empty_like(U), X * Y * Z, _lib.stream_ptr()
    _lib.call("me_sense_forward_volumes", pb.ref, ptr(U), V, 0, S, ptr(K), st)
    _lib.call("me_sense_adjoint_volumes", pb.ref, ptr(K), 0, S, ptr(W), V, st)
    m = pb.mps.to(torch.complex128)
    k = K.reshape(S, Z, C, n).to(torch.complex128)
    e = []
    for s in range(S):
        j = slice(s * n, (s + 1) * n)
        kx = torch.as_tensor(pb.samples.kx[j]).cuda().long()
        ky = torch.as_tensor(pb.samples.ky[j]).cuda().long()
        f = torch.fft.fft2(m * U[s].to(torch.complex128)[:, None], norm="ortho")[..., kx, ky]
        full = torch.zeros((Z, C, X, Y), dtype=torch.complex128, device="cuda")
        full[..., kx, ky] = k[s]
        w = (m.conj() * torch.fft.ifft2(full, norm="ortho")).sum(1)
        e += [float((k[s] - f).norm() / f.norm()), float((W[s] - w).norm() / w.norm())]
    out["sense"].append(e)
    out["stats"].append(pb.lm_stats(rnd(Z, X, Y), 0).cpu().numpy().ravel().tolist())
print(json.dumps(out))
"""


def _run(env):
    r = subprocess.run([sys.executable, "-c", _CHILD, str(ROOT)], env=dict(os.environ, **env),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_stockham_kernels():
    a, b = _run({"ME_GENERIC_FFT": "1"}), _run({})
    assert max(max(e) for e in a["transforms"]) < 2e-6, a["transforms"]
    assert max(max(e) for e in a["sense"]) < 1e-6, a["sense"]
    for x, y in zip(a["stats"], b["stats"]):
        assert max(abs(u - v) for u, v in zip(x, y)) < 1e-5 * max(abs(v) for v in y)
