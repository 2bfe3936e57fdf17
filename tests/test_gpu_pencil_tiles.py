"""The warp-tile pencil beam (dc_pencil.cu) at the sizes where its tiling, spot lists and layer walk can go
wrong, against the CPU oracle: grids one voxel past a tile, more spots than the lists hold, more layers
than a warp tests at once, one and several warps per tile, depth tables that are not evenly spaced.

Tolerance (of the oracle's maximum): positions are rounded to ~1e-5 mm and enter the exponent with
r / sigma^2 < 1 per mm (1e-5), the exponentials hold 2^-22, and a spot beyond 6 sigma_ht (exp(-18) =
1.5e-8 of its peak) is left out, for at most a few hundred spots (1e-5): 2e-5 in all.  Where no spot
comes within the cut-off of any voxel the oracle's maximum itself is such a left-out term; there the dose
only has to vanish."""
import copy
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 2e-5


def _case(shape, n_layers, per_layer, gantry, couch, seed=0, uneven=False, spread=40.0):
    import oracle
    from dosecuda_b200.plan_impt import IMPTPlan
    model = copy.copy(IMPTPlan().beam_models[0])
    if uneven:  # depths 0, 1, 2.001, ...: no even spacing, same range
        d = np.arange(400, dtype=np.float32) * np.linspace(1.0, 1.05, 400, dtype=np.float32)
        model.lut_depths = np.tile(d, (model.lut_depths.shape[0], 1)).astype(np.single)
    rng = np.random.default_rng(seed)
    grid = types.SimpleNamespace(spacing=np.array([2.0, 2.5, 3.0]), origin=np.array([-30.0, -25.0, -20.0]))
    ids = np.linspace(5, 90, n_layers).astype(int) if n_layers > 1 else np.array([40])
    rows = [np.column_stack((rng.uniform(-spread, spread, (per_layer, 2)), rng.uniform(0.5, 1.5, per_layer),
                             np.full(per_layer, e))) for e in ids]
    beam = types.SimpleNamespace(iso=np.array([1.5, -2.0, 3.0], np.single), gantry_angle=gantry, couch_angle=couch,
                                 spot_list=np.vstack(rows).astype(np.single))
    wet = rng.uniform(0.0, 20.0, shape).astype(np.single)
    ref, _ = oracle.proton_dose(wet, grid.spacing, grid.origin, beam.iso, gantry, couch, model, beam.spot_list)
    return model, grid, beam, wet, ref


# 8 x 4 x 4 voxels per warp: one voxel, one full tile, one voxel past a tile on every axis, a slab; spot
# lists of 64 with 1, 64, 65 and 300 spots per layer; 1, 33 and 70 layers
@pytest.mark.parametrize("shape,n_layers,per_layer,gantry,couch,uneven", [
    ((1, 1, 1), 1, 1, 0.0, 0.0, False),
    ((4, 4, 8), 3, 64, 90.0, 0.0, False),
    ((5, 5, 9), 33, 65, 71.7, 20.0, False),
    ((13, 21, 35), 4, 300, 235.0, -30.0, False),
    ((3, 40, 50), 70, 7, 180.0, 0.0, True),
    ((64, 96, 136), 1, 40, 0.0, 0.0, False),   # enough tiles for one warp per tile ...
    ((40, 96, 136), 6, 40, 10.0, 0.0, False),  # ... and for two
])
def test_dose_adjoint_and_list_vs_oracle(shape, n_layers, per_layer, gantry, couch, uneven):
    from dosecuda_b200 import engine
    model, grid, beam, wet, ref = _case(shape, n_layers, per_layer, gantry, couch, uneven=uneven)
    dmax = ref.max()
    assert dmax > 0
    if dmax < 1e-10:  # all spots beyond the cut-off: any dose below this counts as none
        dmax = 1e-10 / TOL
    w = torch.as_tensor(wet, device="cuda")
    dose = engine.proton_dose(w, grid, beam, engine.ProtonModelDevice(model)).cpu().numpy()
    assert np.abs(dose - ref).max() <= TOL * dmax
    plan = engine.ProtonBeamPlan(grid, beam, model)
    assert np.array_equal(plan.dose(w).cpu().numpy(), dose)
    # a list with gaps, repeats and entries outside the grid
    n = wet.size
    vox = np.concatenate((np.arange(0, n, 3), [n - 1, n - 1, -5, n, n + 7])).astype(np.int32)
    out = plan.dose_list(w, torch.as_tensor(vox)).cpu().numpy()
    inside = (vox >= 0) & (vox < n)
    assert np.abs(out[inside] - ref.ravel()[vox[inside]]).max() <= TOL * dmax and (out[~inside] == 0).all()
    # adjoint: g = one voxel's indicator gives that voxel's influence row, whose dot with mu is its dose
    g = np.zeros(shape, np.single)
    hot = np.unravel_index(int(ref.argmax()), shape)
    g[hot] = 1.0
    mu = torch.as_tensor(beam.spot_list[:, 2].astype(np.float64), device="cuda")
    adj = plan.adjoint(w, torch.as_tensor(g, device="cuda"))
    assert abs(float(adj @ mu) - ref[hot]) <= TOL * dmax
    # and <g, D mu> = <D^T g, mu> for a dense g, through the volume and through the list
    g = np.random.default_rng(1).uniform(0.1, 1.0, shape).astype(np.single)
    want = float((g.astype(np.float64) * ref).sum())
    assert abs(float(plan.adjoint(w, torch.as_tensor(g, device="cuda")) @ mu) - want) <= TOL * want
    sel = vox[inside]
    adj = plan.adjoint_list(w, torch.as_tensor(vox), torch.as_tensor(np.where(inside, g.ravel()[np.clip(vox, 0, n - 1)], 7.0)))
    want = float((g.ravel()[sel].astype(np.float64) * ref.ravel()[sel]).sum())
    assert abs(float(adj @ mu) - want) <= TOL * max(want, dmax)


def test_batch_equals_the_one_beam_sum_in_every_variant():
    from dosecuda_b200 import engine
    parts = [_case((13, 21, 35), 4, 100, 30.0, 0.0, seed=1), _case((5, 9, 17), 40, 20, 200.0, 15.0, seed=2)]
    b = engine.ProtonBatch(parts[0][0])
    for model, grid, beam, wet, ref in parts:
        pid = b.add_plan(grid, torch.ones(wet.shape, device="cuda"))
        b.add_beam(pid, beam)
    b.commit()
    for i, p in enumerate(parts):
        b.wets[i].copy_(torch.as_tensor(p[3]))
    for v in range(b.n_variants):
        for d, p in zip(b.dose(variant=v), parts):
            assert np.abs(d.cpu().numpy() - p[4]).max() <= TOL * p[4].max()


def test_spot_positions_that_are_not_finite():
    """A spot at NaN or infinity makes the dose NaN in every voxel its layer reaches, however far the voxel's
    tile is from the layer's other spots (here up to 370 mm)."""
    from dosecuda_b200 import engine
    model, grid, beam, wet, ref = _case((5, 9, 200), 3, 20, 30.0, 0.0, spread=8.0)
    deep = 1.1 * float(model.divergence_params[int(beam.spot_list[0, 3]), 1])
    for bad in (np.nan, np.inf):
        spots = beam.spot_list.copy()
        spots[0, 0] = bad
        dose = engine.proton_dose(torch.as_tensor(wet, device="cuda"), grid, beam, engine.ProtonModelDevice(model),
                                  spots=spots).cpu().numpy()
        assert np.array_equal(np.isnan(dose), (wet * np.float32(10.0)) <= np.float32(deep))


def test_depth_of_minus_infinity():
    """At WET -infinity the air sigma is infinite: the voxel's dose is 0, its neighbours' doses are as they are
    without it."""
    from dosecuda_b200 import engine
    model, grid, beam, wet, ref = _case((9, 13, 40), 3, 20, 30.0, 0.0, spread=8.0)
    wet[4, 6, 20] = -np.inf
    plan = engine.ProtonBeamPlan(grid, beam, model)
    every = torch.arange(wet.size, dtype=torch.int32)
    for dose in (plan.dose(torch.as_tensor(wet, device="cuda")),
                 plan.dose_list(torch.as_tensor(wet, device="cuda"), every).view(wet.shape)):
        dose = dose.cpu().numpy()
        assert dose[4, 6, 20] == 0.0
        dose[4, 6, 20] = ref[4, 6, 20]
        assert np.abs(dose - ref).max() <= TOL * ref.max()


@pytest.mark.parametrize("shape", [(16, 24, 40), (15, 22, 37)])  # full tiles, and tiles with lanes without a voxel
def test_halo_far_from_the_primary(shape):
    """One spot in a smooth depth: most of the volume is reached by its halo alone, whose dose is compared
    relative to itself, down to 1e-6 of the maximum.  There the exponent is at most 14: sigma_h to 4.6e-7 and the
    product's rounding move it by 8e-6, positions to 1e-5 mm by 1e-5 r / sigma_h^2 = 3e-6, exp2 itself 2^-22."""
    import oracle
    from dosecuda_b200 import engine
    model, grid, beam, _, _ = _case((1, 1, 1), 2, 1, 0.0, 0.0)
    beam.spot_list[:, :2] = 4.0, -3.0
    beam.spot_list[:, 3] = 60.0, 75.0
    k, j, i = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    wet = (3.0 + 0.2 * j + 0.01 * i - 0.02 * k).astype(np.single)
    ref, _ = oracle.proton_dose(wet, grid.spacing, grid.origin, beam.iso, 0.0, 0.0, model, beam.spot_list)
    w = torch.as_tensor(wet, device="cuda")
    plan = engine.ProtonBeamPlan(grid, beam, model)
    seen = ref > 1e-6 * ref.max()
    assert 0.5 < seen.mean()
    for dose in (plan.dose(w), plan.dose_list(w, torch.arange(wet.size, dtype=torch.int32)).view(shape)):
        assert np.abs(dose.cpu().numpy() / ref - 1.0)[seen].max() <= 1.2e-5
    mu = torch.as_tensor(beam.spot_list[:, 2].astype(np.float64), device="cuda")
    far = (ref < 1e-3 * ref.max()) & seen  # the adjoint of a gradient on the halo's voxels only
    got = float(plan.adjoint(w, torch.as_tensor(far.astype(np.single), device="cuda")) @ mu)
    assert abs(got / ref[far].sum() - 1.0) <= 1.2e-5


def test_listed_voxels_in_other_company():
    """A listed voxel's dose in lists of another order, length and neighbourhood: its warp's cut-offs may leave out
    other terms, below exp(-18) of a halo peak per spot (all 6 x 40 spots: 240 x 1.5e-8 x the largest halo
    peak, itself below a tenth of the largest dose per spot, which is below the maximum), and its spots are added
    in another order (2^-22 of the dose): 6e-7 of the maximum."""
    from dosecuda_b200 import engine
    model, grid, beam, _, _ = _case((1, 1, 1), 6, 40, 25.0, 10.0)
    shape = (24, 28, 40)
    k, j, i = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    wet = torch.as_tensor((2.0 + 0.25 * j + 0.02 * i - 0.03 * k).astype(np.single), device="cuda")
    plan = engine.ProtonBeamPlan(grid, beam, model)
    n = wet.numel()
    base = plan.dose_list(wet, torch.arange(n, dtype=torch.int32)).cpu().numpy()
    rng = np.random.default_rng(6)
    for pick in (rng.permutation(n), np.arange(n)[::-1], np.arange(0, n, 5), np.sort(rng.choice(n, 700, replace=False))):
        dose = plan.dose_list(wet, torch.as_tensor(pick.astype(np.int32).copy())).cpu().numpy()
        assert np.abs(dose - base[pick]).max() <= 6e-7 * base.max()
