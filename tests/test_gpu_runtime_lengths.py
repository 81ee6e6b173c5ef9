"""Line lengths without a compile-time plan, on the run-time two-stage FFT (fft_rt.cuh), against
the FP64 oracle: every radix in both stages, the smallest lengths, odd lengths, tiles with a
remainder, both volume layouts, all pass modes, and the SENSE kernels at row counts, sample
counts and coil counts that leave remainders.  245 has no such plan and keeps the Stockham
engine.

Tolerances.  One pass rounds each element a dozen times (two FFTs of two stages and the chirp):
about 1.3e-7 relative L2 measured on compile-time lengths, so ten passes give about 4e-7 and
2e-6 is a bound with room, as in test_gpu_transform.py.  SENSE operators: 2e-5 as in
test_gpu_solvers.py."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import Oracle, transform_grids

pytestmark = pytest.mark.gpu

O64 = Oracle(np.complex128)


@pytest.fixture(scope="module")
def me():
    import motionest
    return motionest


def _rnd(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


# per tuple three lengths, each along every axis: all radices up to 32, lengths 1 to 15, odd ones
SHAPES = [(1, 2, 3), (5, 7, 9), (10, 11, 12), (13, 14, 15), (18, 20, 21), (22, 25, 26),
          (27, 28, 30), (33, 35, 39), (42, 45, 49), (50, 65, 77), (84, 90, 91)]


@pytest.mark.parametrize("shape", SHAPES)
def test_transforms(me, shape):
    for turn in range(3):
        sh = tuple(int(n) for n in np.roll(shape, turn))
        rng = np.random.default_rng(sum(sh) + turn)
        x = _rnd(rng, sh)
        kg, rk = transform_grids(sh, [1, 1, 1])
        p = np.array([0.7, -1.1, 0.4, 0.06, -0.05, 0.08])
        T = me.RigidTransformCudaOptimzied(p, kg, rk)
        assert rel_l2(T.apply(x), O64.rigid_apply(x, p, kg, rk)) < 2e-6
        assert rel_l2(T.adjoint(x), O64.rigid_adjoint(x, p, kg, rk)) < 2e-6


@pytest.mark.parametrize("n", [99, 100, 110, 117, 121, 125, 130, 143, 150, 162, 169, 175, 180, 189,
                               198, 200, 208, 216, 220, 225, 231, 234, 240, 242, 243, 245, 250,
                               252, 270, 300, 338, 352, 400, 512])
def test_long_lines(me, n):
    """Long lines as the strided and as the contiguous axis, 21 lines per row (a remainder for
    tiles of 16 and of 8)."""
    for sh in ((n, 3, 7), (3, n, 7), (3, 7, n)):
        rng = np.random.default_rng(n)
        x = _rnd(rng, sh)
        kg, rk = transform_grids(sh, [1, 1, 1])
        p = np.array([-0.6, 0.9, 1.2, -0.04, 0.07, 0.05])
        T = me.RigidTransformCudaOptimzied(p, kg, rk)
        assert rel_l2(T.apply(x), O64.rigid_apply(x, p, kg, rk)) < 2e-6


@pytest.mark.parametrize("shape", [(30, 21, 10), (20, 100, 18), (54, 15, 25), (7, 40, 27)])
@pytest.mark.parametrize("mode", ["reference", "exact"])
def test_partials(me, shape, mode):
    """The dual-output and dual-input passes, one partial at a time and all in one sweep.  A
    partial is a sum of products whose terms are up to about ten times its own size."""
    rng = np.random.default_rng(3)
    x = _rnd(rng, shape)
    kg, rk = transform_grids(shape, [1, 1, 1])
    p = np.array([0.5, -0.3, 0.8, 0.05, -0.06, 0.04])
    D = me.RigidTransformDerivativeCuda(shape, p, kg, rk, jacobian=mode)
    J = D.jacobian(x)
    assert rel_l2(J[0], O64.rigid_apply(x, p, kg, rk)) < 2e-6
    for q in range(6):
        want = O64.rigid_derivative(x, p, q, kg, rk, mode)
        assert rel_l2(D.apply(x, q), want) < 2e-5
        assert rel_l2(J[1 + q], want) < 2e-5


@pytest.mark.parametrize("n", [1, 6, 15, 90, 150, 200, 243, 245])
def test_plain_fft(me, n):
    from motionest.problem import fft_axes
    for axis, sh in enumerate(((n, 5, 4), (5, n, 4), (5, 4, n))):
        x = _rnd(np.random.default_rng(n), (2,) + sh)
        xd = torch.as_tensor(x).cuda()
        f = fft_axes(xd, (axis,), False).cpu().numpy()
        want = np.fft.fft(x.astype(np.complex128), axis=1 + axis, norm="ortho")
        assert rel_l2(f, want) < 1e-6
        back = fft_axes(torch.as_tensor(f).cuda(), (axis,), True).cpu().numpy()
        assert rel_l2(back, x) < 1e-6


# (X, Y), coils, shots, sampled share: rows per CTA 32, 24, 16 and 8, X with a remainder, one and
# several samples per thread, a Y whose second radix is large, an empty shot
SENSE = [((21, 10), 3, 3, 0.4), ((50, 49), 5, 3, 0.3), ((35, 84), 2, 4, 0.2), ((33, 100), 3, 2, 0.5),
         ((70, 150), 2, 5, 0.1), ((40, 150), 9, 3, 0.3), ((30, 200), 2, 3, 0.2),
         ((18, 243), 2, 3, 0.05), ((9, 30), 3, 1, 1.0), ((11, 245), 2, 2, 0.1)]


@pytest.mark.parametrize("xy,coils,shots,share", SENSE)
def test_sense(me, xy, coils, shots, share):
    from motionest.problem import SenseProblem, xyz_to_zxy, zxy_to_xyz
    shape = xy + (3,)
    rng = np.random.default_rng(sum(xy))
    planes = rng.random((shots,) + xy) < share
    if shots > 2:
        planes[1] = False
    mps, ksp, x = 0.5 * _rnd(rng, (coils,) + shape), _rnd(rng, (coils,) + shape), _rnd(rng, shape)
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
    e = pb.residual_norms(xd, pb.transforms).cpu().numpy()
    st = pb.lm_stats(xd, 0).cpu().numpy()
    for s in range(shots):
        r = O64.forward_residual(ksp, mps, mask[s], x, t[s], kg, rk)
        want = O64.vdot_real(r, r)
        np.testing.assert_allclose(e[s], want, rtol=1e-5, atol=1e-12)
        np.testing.assert_allclose(st[s, 0], want, rtol=1e-5, atol=1e-12)
        J = O64.jacobian(ksp.shape, mps, mask[s], x, t[s], kg, rk)
        g = np.array([O64.vdot_real(r, j) for j in J])
        n = np.sqrt(want * np.array([O64.vdot_real(j, j) for j in J]))
        assert np.all(np.abs(st[s, 1:7] - g) <= 2e-5 * n + 1e-12)
