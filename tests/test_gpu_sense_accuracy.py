"""Rounding of the SENSE kernels alone (me_sense_forward_volumes,
me_sense_adjoint_volumes), against the same model by torch
FFTs in complex128: tolerances of a few units in the last place, which the looser parity tests
cannot stand in for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

Z, S = 2, 3


def _problem(X, Y, C, seed):
    from motionest.problem import SenseProblem
    from motionest.utils import compute_transform_grids_voxel
    rng = np.random.default_rng(seed)
    n = min(X * Y // 3, 400)
    planes = np.zeros((S, X * Y), bool)
    for s in range(S):
        planes[s, rng.choice(X * Y, n, replace=False)] = True
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*shape):
        return torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g)

    kg, rk = compute_transform_grids_voxel((X, Y, Z), [1, 1, 1])
    t = torch.zeros((S, 6), dtype=torch.float64, device="cuda")
    mps = rnd(C, X, Y, Z)
    return SenseProblem(None, mps, planes.reshape(S, X, Y), kg, rk, t), rnd, n


def _shots(pb, n):
    for s in range(S):
        j = slice(s * n, (s + 1) * n)
        yield s, (torch.as_tensor(pb.samples.kx[j]).cuda().long(),
                  torch.as_tensor(pb.samples.ky[j]).cuda().long())


def _rel(got, ref):
    return float(torch.linalg.vector_norm(got - ref) / torch.linalg.vector_norm(ref))


@pytest.mark.parametrize("Y", [48, 72, 88, 96, 112, 128, 224, 90, 150])
@pytest.mark.parametrize("X", [37, 128, 256])
def test_forward_against_fp64(X, Y):
    """Relative L2 below 2.0e-7.  The sums along x in float32, Horner chains of eight rows with one
    table twiddle a chain, round to 1.2 to 1.3e-7 (emulated in numpy, fused multiply-adds); the FFT
    along y and the product with the maps add about 1.1e-7 in quadrature (two roundings in each
    of some log2(Y) + 2 levels, 3e-8 each).  Chains of sixteen rows alone round to 1.9 to 2.3e-7."""
    from motionest import _lib
    from motionest._lib import ptr
    C = 4
    pb, rnd, n = _problem(X, Y, C, 1000 * Y + X)
    U = rnd(S, Z, X, Y)
    K = torch.empty(S * n * C * Z, dtype=torch.complex64, device="cuda")
    _lib.call("me_sense_forward_volumes", pb.ref, ptr(U), X * Y * Z, 0, S, ptr(K),
              _lib.stream_ptr())
    m = pb.mps.to(torch.complex128)
    ref = torch.stack([torch.fft.fft2(m * U[s].to(torch.complex128)[:, None], norm="ortho")[..., kx, ky]
                       for s, (kx, ky) in _shots(pb, n)])
    assert _rel(K.reshape(ref.shape).to(torch.complex128), ref) < 2.0e-7


@pytest.mark.parametrize("Y", [48, 64, 72, 88, 96, 112, 128, 256, 40, 80, 90, 150, 160, 200])
@pytest.mark.parametrize("X", [128, 150])
def test_adjoint_against_fp64(X, Y):
    """Relative L2 below 1.75e-7 with 32 coils.  One rounding a coil (2.5e-8 of the running sum, which
    grows with the root of the coils) makes 1.0e-7 of the sum over the coils; the walk along x
    (6.4e-8 emulated), the FFT along y and the products make about 1.25e-7: together 1.6e-7.
    Two roundings a coil make 1.4e-7 of the sum and 1.9e-7 of all."""
    from motionest import _lib
    from motionest._lib import ptr
    C = 32
    pb, rnd, n = _problem(X, Y, C, 1000 * Y + X)
    K = rnd(S * n * C * Z)
    W = torch.empty((S, Z, X, Y), dtype=torch.complex64, device="cuda")
    _lib.call("me_sense_adjoint_volumes", pb.ref, ptr(K), 0, S, ptr(W), X * Y * Z,
              _lib.stream_ptr())
    m = pb.mps.to(torch.complex128)
    ref = torch.empty((S, Z, X, Y), dtype=torch.complex128, device="cuda")
    for s, (kx, ky) in _shots(pb, n):
        full = torch.zeros((Z, C, X, Y), dtype=torch.complex128, device="cuda")
        full[..., kx, ky] = K[s * n * C * Z:(s + 1) * n * C * Z].reshape(Z, C, n).to(full.dtype)
        ref[s] = (m.conj() * torch.fft.ifft2(full, norm="ortho")).sum(1)
    assert _rel(W.to(torch.complex128), ref) < 1.75e-7
