"""SENSE kernels on caller-transformed volumes of more planes than a grid's z extent holds (65,535), at a
width without a compile-time plan: taken, with the same values as plane by plane in complex128."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_planes_than_a_grid_is_deep():
    from motionest import _lib
    from motionest._lib import ptr
    from motionest.problem import SenseProblem
    from motionest.utils import compute_transform_grids_voxel
    X, Y, Z, C = 2, 3, 65537, 1
    planes = np.zeros((1, X, Y), bool)
    planes[0, 0, 1] = planes[0, 1, 2] = True
    g = torch.Generator(device="cuda").manual_seed(2)
    mps = torch.randn((C, X, Y, Z), dtype=torch.complex64, device="cuda", generator=g)
    kg, rk = compute_transform_grids_voxel((X, Y, Z), [1, 1, 1])
    pb = SenseProblem(None, mps, planes, kg, rk,
                      torch.zeros((1, 6), dtype=torch.float64, device="cuda"), lm_batch=1)
    U = torch.randn((Z, X, Y), dtype=torch.complex64, device="cuda", generator=g)
    K, W, st = torch.empty_like(pb.ydat), torch.empty_like(U), _lib.stream_ptr()
    _lib.call("me_sense_forward_volumes", pb.ref, ptr(U), X * Y * Z, 0, 1, ptr(K), st)
    _lib.call("me_sense_adjoint_volumes", pb.ref, ptr(K), 0, 1, ptr(W), X * Y * Z, st)
    m = mps.permute(3, 0, 1, 2).to(torch.complex128)
    F = torch.fft.fft2(m * U[:, None].to(torch.complex128), norm="ortho")
    kx, ky = torch.tensor([0, 1]).cuda(), torch.tensor([1, 2]).cuda()  # by ky
    ref = F[..., kx, ky]
    full = torch.zeros_like(F)
    full[..., kx, ky] = ref
    back = (m.conj() * torch.fft.ifft2(full, norm="ortho")).sum(1)
    # 2- and 3-point transforms: some ten roundings of 6e-8
    assert torch.linalg.vector_norm(K.reshape(ref.shape) - ref) < 6e-7 * torch.linalg.vector_norm(ref)
    assert torch.linalg.vector_norm(W - back) < 1.2e-6 * torch.linalg.vector_norm(back)
