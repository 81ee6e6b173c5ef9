"""Compile-time line lengths beside dimensions that leave remainders, against the FP64 oracle:
strided tiles that end past the row (row lengths 33 to 88 that are no multiples of 16), contiguous
tiles that run over into the next rows or end early, odd rows (no TMA), one-tile launches, and the
SENSE kernels at every kind of row-range plan (row counts, split bins, one to eight samples per
thread).  Tolerances as in test_gpu_transform.py and test_gpu_solvers.py."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import Oracle, transform_grids

pytestmark = pytest.mark.gpu

O64 = Oracle(np.complex128)


def _rnd(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("shape", [(16, 64, 40), (48, 72, 56), (128, 24, 88), (32, 112, 20),
                                   (96, 16, 36), (256, 16, 50), (64, 35, 33), (144, 3, 192),
                                   (2, 176, 224), (128, 1, 64)])
def test_transforms(shape):
    import motionest as me
    rng = np.random.default_rng(sum(shape))
    kg, rk = transform_grids(shape, [1, 1, 1])
    x = _rnd(rng, shape)
    p = np.array([0.7, -1.1, 0.4, 0.06, -0.05, 0.08])
    T = me.RigidTransformCudaOptimzied(p, kg, rk)
    assert rel_l2(T.apply(x), O64.rigid_apply(x, p, kg, rk)) < 2e-6
    assert rel_l2(T.adjoint(x), O64.rigid_adjoint(x, p, kg, rk)) < 2e-6
    J = me.RigidTransformDerivativeCuda(shape, p, kg, rk, jacobian="exact").jacobian(x)
    for q in range(6):
        assert rel_l2(J[1 + q], O64.rigid_derivative(x, p, q, kg, rk, "exact")) < 2e-5


def test_chained_launches_see_earlier_work():
    """Transforms of one small volume chained on a stream, each reading the last one's result and
    parameters written just before it: the same bits as with a synchronisation after each."""
    from motionest.problem import SenseProblem
    shape = (32, 24, 16)
    rng = np.random.default_rng(1)
    kg, rk = transform_grids(shape, [1, 1, 1])
    mps = torch.as_tensor(_rnd(rng, (1,) + shape)).cuda()
    pb = SenseProblem(None, mps, np.ones((1, 32, 24), bool), kg, rk,
                      torch.zeros((1, 6), dtype=torch.float64, device="cuda"))
    x0 = torch.as_tensor(_rnd(rng, (16, 32, 24))).cuda()
    prm = [torch.as_tensor(rng.uniform(-0.2, 0.2, 6)).cuda() for _ in range(6)]
    res = []
    for sync in (True, False):
        x, p = x0.clone(), torch.zeros(6, dtype=torch.float64, device="cuda")
        for q in prm * 4:
            p.copy_(q)
            x = pb.apply_transform(x, p, out=torch.empty_like(x))
            if sync:
                torch.cuda.synchronize()
        res.append(x)
    assert torch.equal(res[0], res[1])


@pytest.mark.parametrize("xy,shots,share", [((20, 16), 2, 0.5), ((33, 24), 2, 0.4), ((40, 48), 3, 0.3),
                                            ((50, 72), 2, 0.5), ((18, 88), 2, 0.4), ((70, 96), 2, 0.2),
                                            ((45, 128), 3, 0.3), ((21, 144), 3, 0.1),
                                            ((20, 176), 2, 0.02), ((35, 192), 2, 0.25),
                                            ((9, 256), 2, 0.8), ((24, 224), 3, 0.05)])
def test_sense(xy, shots, share):
    from motionest.problem import SenseProblem, xyz_to_zxy, zxy_to_xyz
    shape = xy + (2,)
    rng = np.random.default_rng(sum(xy))
    planes = rng.random((shots,) + xy) < share
    mps, ksp, x = 0.5 * _rnd(rng, (3,) + shape), _rnd(rng, (3,) + shape), _rnd(rng, shape)
    t = np.zeros((shots, 6))
    t[:, :3] = rng.uniform(-2, 2, (shots, 3))
    t[:, 3:] = np.deg2rad(rng.uniform(-4, 4, (shots, 3)))
    kg, rk = transform_grids(shape, [1, 1, 1])
    dev = lambda a: torch.as_tensor(a).cuda()  # noqa: E731
    pb = SenseProblem(dev(ksp), dev(mps), planes, kg, rk, dev(t))
    xd = xyz_to_zxy(dev(x))
    mask = planes[..., None]
    M = (np.abs(mps) ** 2).sum(0) > 0.1
    got = zxy_to_xyz(pb.normal(xd, pb.empty_image())).cpu().numpy()
    assert rel_l2(got, O64.normal_op(x, mps, mask, t, kg, rk, M)) < 2e-5
    got = zxy_to_xyz(pb.rhs(pb.empty_image())).cpu().numpy()
    assert rel_l2(got, O64.cg_rhs(ksp, mps, mask, t, kg, rk, M)) < 2e-5
    st = pb.lm_stats(xd, 0).cpu().numpy()
    for s in range(shots):
        r = O64.forward_residual(ksp, mps, mask[s], x, t[s], kg, rk)
        J = O64.jacobian(ksp.shape, mps, mask[s], x, t[s], kg, rk)
        n = np.sqrt(O64.vdot_real(r, r) * np.array([O64.vdot_real(j, j) for j in J]))
        g = np.array([O64.vdot_real(r, j) for j in J])
        np.testing.assert_allclose(st[s, 0], O64.vdot_real(r, r), rtol=1e-5)
        assert np.all(np.abs(st[s, 1:7] - g) <= 2e-5 * n)
