"""Memory of the motion step's workspace: the default number of shots a launch gives way where the
device is short of memory, a forward-only problem takes none, and the batch does not change the
statistics."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(nshots=64, **kw):
    from motionest.problem import SenseProblem
    from motionest.utils import compute_transform_grids_voxel
    shape, C = (64, 60, 24), 2
    rng = np.random.default_rng(0)
    planes = rng.random((nshots,) + shape[:2]) < 0.05
    mps = torch.as_tensor((rng.standard_normal((C,) + shape)
                           + 1j * rng.standard_normal((C,) + shape)).astype(np.complex64)).cuda()
    kg, rk = compute_transform_grids_voxel(shape, [1, 1, 1])
    t = torch.as_tensor(rng.uniform(-0.05, 0.05, (nshots, 6))).cuda()
    return SenseProblem(mps.clone(), mps, planes, kg, rk, t, **kw)


def test_default_batch_follows_free_memory(monkeypatch):
    total = torch.cuda.mem_get_info()[1]
    full = _problem()
    assert full.lm_batch == 64  # 9 MB a shot
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (1 << 30, total))
    short = _problem()
    assert short.lm_batch == 8
    assert _problem(lm_batch=16).lm_batch == 16  # an explicit one stays
    assert _problem(nshots=16).lm_batch == 16    # and a few MB more are not asked for
    x = torch.randn((24, 64, 60), dtype=torch.complex64, device="cuda")
    assert torch.equal(full.lm_stats(x, 0), short.lm_stats(x, 0))


def test_simulation_takes_no_motion_workspace(monkeypatch):
    from motionest import simulation
    made = []

    class Problem(simulation.SenseProblem):
        def __init__(self, *a, **kw):
            super().__init__(*a, **kw)
            made.append(self)

    monkeypatch.setattr(simulation, "SenseProblem", Problem)
    shape, S = (32, 30, 12), 16
    img = simulation.phantom(shape, 4, 0, "cuda")
    mps = simulation.coil_maps(shape, 2, 0, device="cuda")
    from motionest.sampling import disorder_masks
    masks = disorder_masks(32, 30, (4, 3), 1, S)
    simulation.generate_corrupted_kspace(img, mps, masks, np.zeros((S, 6)))
    assert made and made[0].lm_batch == 1
