"""Rounding of the SENSE kernels alone (me_sense_forward_volumes), against the same model by torch
FFTs in complex128: tolerances of a few units in the last place, which the looser parity tests
cannot stand in for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

C, Z, S = 4, 2, 3


def _problem(X, Y, seed):
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
    pb, rnd, n = _problem(X, Y, 1000 * Y + X)
    U = rnd(S, Z, X, Y)
    K = torch.empty(S * n * C * Z, dtype=torch.complex64, device="cuda")
    _lib.call("me_sense_forward_volumes", pb.ref, ptr(U), X * Y * Z, 0, S, ptr(K),
              _lib.stream_ptr())
    m = pb.mps.to(torch.complex128)
    ref = torch.stack([torch.fft.fft2(m * U[s].to(torch.complex128)[:, None], norm="ortho")[..., kx, ky]
                       for s, (kx, ky) in _shots(pb, n)])
    assert _rel(K.reshape(ref.shape).to(torch.complex128), ref) < 2.0e-7
