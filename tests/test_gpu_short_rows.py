"""Strided tiles of rows of 16 to 31 lines (a full tile and one of 2 to 15 lines) on the tensor-map
kernel, all pass modes, against the FP64 oracle, and beside the same volume 8 bytes off a 16-byte
boundary, which the cp.async kernel takes with the same bits.  Tolerances as in
test_gpu_ragged_tiles.py."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import Oracle, transform_grids

pytestmark = pytest.mark.gpu

O64 = Oracle(np.complex128)


@pytest.mark.parametrize("shape", [(64, 48, 18), (32, 24, 20), (128, 16, 22), (16, 56, 24),
                                   (88, 112, 26), (48, 144, 28), (224, 32, 30), (24, 32, 15)])
def test_rows_of_less_than_two_tiles(shape):
    import motionest as me
    from motionest import _lib
    from motionest.utils import device_grid
    rng = np.random.default_rng(sum(shape))
    kg, rk = transform_grids(shape, [1, 1, 1])
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    p = np.array([0.7, -1.1, 0.4, 0.06, -0.05, 0.08])
    T = me.RigidTransformCudaOptimzied(p, kg, rk)
    assert rel_l2(T.apply(x), O64.rigid_apply(x, p, kg, rk)) < 2e-6
    assert rel_l2(T.adjoint(x), O64.rigid_adjoint(x, p, kg, rk)) < 2e-6
    J = me.RigidTransformDerivativeCuda(shape, p, kg, rk, jacobian="exact").jacobian(x)
    for q in range(6):
        assert rel_l2(J[1 + q], O64.rigid_derivative(x, p, q, kg, rk, "exact")) < 2e-5
    n = x.size
    prm = torch.as_tensor(p).cuda()
    outs = []
    for off in (0, 1):
        src = torch.zeros(n + 2, dtype=torch.complex64, device="cuda")[off:off + n]
        dst = torch.zeros(n + 2, dtype=torch.complex64, device="cuda")[off:off + n]
        src.copy_(torch.as_tensor(x.ravel()))
        _lib.call("me_rigid_apply", _lib.ptr(src), 0, _lib.ptr(dst), 0, 1,
                  _lib.MeLayout(shape[1] * shape[2], shape[2], 1), device_grid(kg, rk, shape).ref,
                  _lib.ptr(prm), 0, 0, _lib.stream_ptr())
        outs.append(dst.cpu())
    assert torch.equal(outs[0], outs[1])
    assert _lib.wait_status() == 0
