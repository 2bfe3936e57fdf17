"""The tiled collapsed-cone kernel (dc_cccs.cu) where its split of the samples between the texture unit and
shared memory, its tiles and its voxel mask can go wrong, against the CPU oracle with the texture unit's
rounded axis fractions: grids one voxel past a tile, spacings that put 1 to 10 samples of a cone in shared
memory, uneven spacings, fields that leave tiles partly or wholly masked.

Tolerance: the oracle rounds the three fractions to 1/256 and multiplies them exactly; the hardware also
rounds each of the eight products to 1/256 (half a unit, 1/512, each way).  A sample between texels that
differ by the whole range (a material boundary, the field's edge) is then off by up to 1/512 of it; over the
hundreds of samples of a voxel these average out by more than 3: 1e-3 of the dose maximum.  Voxels whose
TERMA lies within 1 % of the mask's threshold are left out: there both sides are right, dose or none."""
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing,gantry,couch,field", [
    ((5, 9, 9), (2.5, 2.5, 2.5), 0.0, 0.0, 30.0),       # one voxel past a tile
    ((1, 1, 40), (2.0, 2.0, 2.0), 90.0, 0.0, 20.0),     # a single row
    ((30, 33, 41), (4.0, 4.0, 4.0), 37.0, 15.0, 60.0),  # few samples per cone
    ((24, 30, 28), (1.0, 1.0, 1.0), 200.0, 0.0, 12.0),  # many
    ((33, 40, 47), (2.5, 2.0, 3.0), 310.0, -20.0, 40.0),  # uneven spacings: the reach differs per axis
    ((70, 90, 97), (3.0, 3.0, 3.0), 25.0, 0.0, 50.0),   # most tiles masked
])
def test_dose_vs_oracle(shape, spacing, gantry, couch, field):
    import oracle
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    rng = np.random.default_rng(sum(shape))
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array(spacing), origin=np.array([-n * s / 2 for n, s in zip((nx, ny, nz), spacing)]))
    rho = np.ones(shape, np.single)
    rho += 0.02 * rng.standard_normal(shape).astype(np.single)
    rho[: nz // 3, : ny // 2, : nx // 2] = 0.3
    x12 = np.where(np.abs(model.mlc_offsets) <= field / 2 + 5, field / 2, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.array([0.7, -1.1, 0.4], np.single), 100.0, mlc, gantry, 10.0, couch, None, None)
    vol = torch.as_tensor(rho, device="cuda")
    was = engine.photon_depth_mode(0)
    engine.photon_depth_mode(0, "march")  # the reference's depth, so that only the superposition differs
    try:
        _check(engine, oracle, vol, rho, grid, spacing, model, cp, rng)
    finally:
        engine.photon_depth_mode(0, was)


def _check(engine, oracle, vol, rho, grid, spacing, model, cp, rng):
    dose = engine.photon_dose(vol, grid, model, cp).cpu().numpy()
    ref, terma, _, _ = oracle.photon_dose(rho, spacing, grid.origin, model, cp.iso, cp.mu, cp.ga, cp.ca, cp.ta,
                                          np.ascontiguousarray(cp.mlc), tex_mode=1, intermediates=True)
    assert ref.max() > 0
    sure = np.abs(terma - 0.01) > 1e-4  # the mask drops the whole dose of a voxel at TERMA 0.01
    assert sure.mean() > 0.99
    assert np.abs(dose - ref)[sure].max() <= 1e-3 * ref.max()
    # the same voxels through the probe's mask
    beam = engine.PhotonBeam(grid, rho.shape)
    beam.set_density(vol)
    beam.terma(model, cp)
    pick = np.concatenate((rng.integers(0, rho.size, 50), [-1, rho.size])).astype(np.int32)
    got = beam.probe(torch.as_tensor(pick, device="cuda")).cpu().numpy()
    assert np.array_equal(got[:-2], dose.ravel()[pick[:-2]]) and (got[-2:] == 0).all()
    beam.close()


@pytest.mark.parametrize("shape,spacing,field,lists", [
    ((40, 44, 52), (2.5, 2.5, 2.5), 40.0, ("all", "third", "shuffled")),   # a box per voxel, shared boxes
    ((24, 30, 40), (1.0, 1.0, 1.0), 15.0, ("all", "third", "shuffled")),   # boxes too large for four per block
    ((3, 70, 300), (2.0, 2.0, 2.0), 60.0, ("all", "third")),               # rows longer than a run, runs across rows
    ((70, 60, 64), (3.0, 2.0, 2.5), 80.0, ("all",)),                       # more entries per block
])
def test_lists_equal_the_full_dose(shape, spacing, field, lists):
    """A probe's dose is the full calculation's bit for bit, whichever way its list is worked through: every
    voxel and every third in order, in any order with repeats, with entries outside the grid."""
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    rng = np.random.default_rng(sum(shape))
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array(spacing), origin=np.array([-n * s / 2 for n, s in zip((nx, ny, nz), spacing)]))
    x12 = np.where(np.abs(model.mlc_offsets) <= field / 2, field / 2, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, 33.0, 0.0, 20.0, None, None)
    beam = engine.PhotonBeam(grid, shape)
    beam.set_density(torch.as_tensor(rng.uniform(0.2, 1.6, shape).astype(np.single), device="cuda"))
    beam.terma(model, cp)
    full = beam.dose().reshape(-1)
    n = full.numel()
    assert bool((full > 0).any()) and bool((full == 0).any())
    for kind in lists:
        pick = {"all": np.arange(n), "third": np.arange(1, n, 3), "shuffled": rng.integers(0, n, n)}[kind].astype(np.int32)
        out = rng.integers(0, pick.size, 20)
        pick[out[:10]], pick[out[10:]] = -1, n
        v = torch.as_tensor(pick, device="cuda").long()
        want = torch.where((v >= 0) & (v < n), full[v.clamp(0, n - 1)], torch.zeros((), device="cuda"))
        for part in (pick.size, 5000):  # long and short
            got = beam.probe(torch.as_tensor(pick[:part], device="cuda"))
            assert torch.equal(got, want[:part])
    beam.close()
