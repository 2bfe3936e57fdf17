"""The fluence adjoint's scatter (dc_fluence.cu: pairs of voxels per 16-byte addition) on grids where pairs end
at the volume's edge: one voxel along an axis, odd and even extents."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 9, 2), (3, 5, 7), (6, 1, 33), (4, 8, 6)])
def test_dose_and_adjoint_agree(shape):
    """<g, dose(F)> = <adjoint(g), F>.  The dose's texture weights are rounded to 1/256 (half a unit, 1/512,
    either way) while the adjoint's are not; on these grids most samples blend with the border's 0, so that
    a sample may be off by 1/512 of itself: 2e-3 of the sum of |g| dose.  One voxel's part of the sum lost
    or added elsewhere is larger than that."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    nz, ny, nx = shape
    sp = 4.0
    grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([-n * sp / 2 for n in (nx, ny, nz)]))
    rho = torch.ones(shape, device="cuda")
    x12 = np.where(np.abs(model.mlc_offsets) <= 100.0, 90.0, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.array([0.0, 0.0, 0.0], np.single), 100.0, mlc, 30.0, 0.0, 15.0, None, None)
    fb = engine.PhotonFluenceBeam.field_map(rho, grid, model, cp, pitch=30.0, margin=10.0)
    gen = torch.Generator().manual_seed(2)
    F = (torch.rand((fb.nb, fb.na), generator=gen) + 0.5).cuda()
    dose = fb.dose(F).double()
    for _ in range(4):
        g = torch.randn(shape, generator=gen).cuda()
        lhs, rhs = float((g.double() * dose).sum()), float((fb.adjoint(g).reshape(F.shape) * F.double()).sum())
        assert abs(lhs - rhs) <= 2e-3 * float((g.double().abs() * dose).sum())


def test_probe_after_a_fluence_dose():
    """The probe leaves out voxels by their TERMA as it is in the beam: where the map is 0 it gives 0, although the
    dose there, masked by the unmodulated TERMA, holds scatter from the open half.  Elsewhere both agree."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    shape, sp = (24, 20, 28), 3.0
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([-n * sp / 2 for n in (nx, ny, nz)]))
    x12 = np.where(np.abs(model.mlc_offsets) <= 30.0, 30.0, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, 0.0, 0.0, 0.0, None, None)
    fb = engine.PhotonFluenceBeam.field_map(torch.ones(shape, device="cuda"), grid, model, cp, pitch=5.0)
    F = torch.ones((fb.nb, fb.na), device="cuda")
    F[:, : fb.na // 2] = 0.0
    dose = fb.dose(F).reshape(-1)
    probe = fb.beam.probe(torch.arange(dose.numel(), device="cuda", dtype=torch.int32))
    kept = probe != 0
    assert torch.equal(probe[kept], dose[kept])
    left_out = (dose > 1e-3 * dose.max()) & ~kept  # scatter under the closed half
    assert 20 <= int(left_out.sum()) < int(kept.sum())


def test_adjoint_of_an_infinite_gradient():
    """An infinite gradient at one voxel makes the beamlets infinite that its dose depends on, and none NaN: texels
    with weight 0 take no part of it, and no part of a sample is a difference of infinities.  The voxel lies at
    the surface, where TERMA and the electron term of all texels in reach are above 0."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    shape, sp = (9, 6, 10), 4.0
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([-n * sp / 2 for n in (nx, ny, nz)]))
    x12 = np.where(np.abs(model.mlc_offsets) <= 100.0, 90.0, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, 0.0, 0.0, 0.0, None, None)
    fb = engine.PhotonFluenceBeam.field_map(torch.ones(shape, device="cuda"), grid, model, cp, pitch=5.0)
    for at in ((4, 0, 5), (0, 2, 0), (8, 3, 9)):
        g = torch.zeros(shape, device="cuda")
        g[at] = 1.0
        want = fb.adjoint(g) != 0
        g[at] = float("inf")
        got = fb.adjoint(g)
        assert torch.equal(got == float("inf"), want) and bool((got[~want] == 0).all())
