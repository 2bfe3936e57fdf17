"""How exactly the warp-tile pencil beam (dc_pencil.cu) holds a pair's influence, against float64 on the same
float32 inputs."""
import copy
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _model(sigma, idd, r80):
    """A beam model of n energies whose spot sigma and depth dose are constants: no rounding before the
    Gaussians' norms."""
    from dosecuda_b200.plan_impt import IMPTPlan
    model = copy.copy(IMPTPlan().beam_models[0])
    n = len(r80)
    dvp = np.zeros((n, model.divergence_params.shape[1]), np.single)
    dvp[:, 1] = r80
    model.divergence_params = dvp
    ones = np.ones((n, 400), np.single)
    model.lut_depths = ones * np.arange(400, dtype=np.single)
    model.lut_sigmas = ones * np.asarray(sigma, np.single)[:, None]
    model.lut_idds = ones * np.asarray(idd, np.single)[:, None]
    return model


def _influence64(wet, r80, sigma, idd, r2):
    """Dose per MU at squared axis distance r2, float64 (nuclearHalo and pencilBeamKernel, IMPTClasses.cu:104-121,
    204-271)."""
    w = np.clip((wet * np.float32(10.0)).astype(np.float64), 0.1, r80 - 0.1)
    hs = 2.85 + 0.0014 * r80 * np.log(w + 3) + 0.06 * w - 7.4e-5 * w * w - 0.22 * r80 / (w - r80 - 5) ** 2
    hw = 0.052 * np.log(1.13 + w / (11.2 - 0.023 * r80)) + 0.35 * (0.0017 * r80 ** 2 - r80) / ((r80 + 3) ** 2 - w * w) \
        - 1.61e-9 * w * (r80 + 3) ** 2
    wh, t2 = np.clip(hw, 0.0, 0.9), sigma ** 2
    h2 = t2 + np.maximum(hs, 0.0) ** 2
    return (1 - wh) * idd / (2 * np.pi * t2) * np.exp(-0.5 * r2 / t2) + wh * idd / (2 * np.pi * h2) * np.exp(-0.5 * r2 / h2)


def test_influence_on_the_axis():
    """On a spot's axis the influence is pf + hf.  Rounded to 32 bits with IEEE operations, pf takes three
    roundings after 1 - wh (product with idd, 2 pi sigma^2, quotient), the sum a fourth and 1 - wh a fifth,
    each 2^-24 / sqrt(3) * sqrt(0.541) = 2.5e-8 rms over evenly spread mantissas, and 2 pi itself is off by
    2.8e-8: 6.3e-8 rms.  A sixth rounding makes 6.8e-8; the bound lies between."""
    from dosecuda_b200 import engine
    rng = np.random.default_rng(11)
    n, energies = 4096, 24
    r80 = rng.uniform(40.0, 340.0, energies).astype(np.single)
    sigma = (rng.integers(8, 40, energies) / 4.0).astype(np.single)  # squares exact
    idd = rng.uniform(0.1, 3.0, energies).astype(np.single)
    model = _model(sigma, idd, r80)
    dm = engine.ProtonModelDevice(model)
    grid = types.SimpleNamespace(spacing=np.array([2.0, 0.25, 2.0]), origin=np.array([0.0, -512.0, 0.0]))
    sq = 0.0
    for e in range(energies):
        beam = types.SimpleNamespace(iso=np.zeros(3, np.single), gantry_angle=0.0, couch_angle=0.0,
                                     spot_list=np.array([[0.0, 0.0, 1.0, e]], np.single))
        wet = (rng.uniform(0.02, 0.98, (1, n, 1)) * r80[e] / 10.0).astype(np.single)
        dose = engine.proton_dose(torch.as_tensor(wet, device="cuda"), grid, beam, dm).cpu().numpy()
        ref = _influence64(wet, float(r80[e]), float(sigma[e]), float(idd[e]), 0.0)
        sq += float(((dose / ref - 1.0) ** 2).mean())
    assert (sq / energies) ** 0.5 <= 6.55e-8


def test_listed_voxels_far_from_the_isocentre():
    """A listed voxel's distance from a spot 150 to 190 mm off the isocentre, at most 16 mm: in coordinates
    relative to the spot three roundings and those of the unit vector, 4 x 2^-24 x 16 mm = 4e-6 mm, move
    the Gaussian by r dr / sigma^2 = 16 x 4e-6 / 36 = 2e-6, the exponent's own rounding (5 x 2^-23) by
    6e-7 and the parameters by 1e-6: 4e-6.  Coordinates relative to the isocentre would move it by
    190 / 16 times the first figure, 2e-5."""
    from dosecuda_b200 import engine
    r80, sigma, idd = np.array([120.0], np.single), np.array([6.0], np.single), np.array([1.5], np.single)
    model = _model(sigma, idd, r80)
    shape = (12, 9, 16)  # exact coordinates: gantry 0, powers of two
    sp = 2.0
    rng = np.random.default_rng(3)
    for sx, sy in ((160.0, -152.0), (-184.0, 176.0), (150.5, 188.25)):
        grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([0.0, 0.0, 0.0]))
        # head x, y = -/+ image x, z at gantry 0: the volume lies around the spot's axis
        for fx, fz in ((1, 1), (-1, 1), (1, -1), (-1, -1)):
            iso = np.array([16.0 - fx * sx, 8.0, 12.0 - fz * sy], np.single)
            beam = types.SimpleNamespace(iso=iso, gantry_angle=0.0, couch_angle=0.0,
                                         spot_list=np.array([[sx, sy, 1.0, 0.0]], np.single))
            wet = rng.uniform(0.5, 11.0, shape).astype(np.single)
            w = torch.as_tensor(wet, device="cuda")
            plan = engine.ProtonBeamPlan(grid, beam, model)
            vox = torch.arange(wet.size, device="cuda", dtype=torch.int32)
            dose = plan.dose_list(w, vox).cpu().numpy().reshape(shape)
            k, j, i = np.meshgrid(*[np.arange(m, dtype=np.float64) * sp for m in shape], indexing="ij")
            x, y, z = i - iso[0], j - iso[1], k - iso[2]
            # the frame turns by 180 degrees, with the sine of the float32 pi
            s180 = np.sin(np.float64(np.float32(np.pi)))
            h = np.stack((x - y * s180, z, -x * s180 - y))
            t = np.array([sx / float(model.VSADX), sy / float(model.VSADY), -1.0])
            ray = h - np.array([sx, sy, 0.0])[:, None, None, None]
            cross = np.cross(ray, t, axisa=0, axisc=0)
            r2 = (cross ** 2).sum(0) / (t ** 2).sum()
            near = r2 < 16.0 ** 2
            if not near.any():
                continue
            ref = _influence64(wet, 120.0, 6.0, 1.5, r2)
            assert np.abs(dose / ref - 1.0)[near].max() <= 4e-6
            break
        else:
            raise AssertionError("the volume lies beside the spot")


@pytest.mark.parametrize("step", [0.7, 1.5])
def test_depth_tables_in_decimal_steps(step):
    """Depths q x 0.7 in float32 follow the even spacing bit for bit while their differences do not (up to
    2.6e-5 of the step); a depth dose that goes up and down by a factor of 3 from row to row shows a factor
    past / step instead of past / (difference).  The interpolation takes two roundings (2^-23), the pair's
    influence 3e-7: 1e-6 in all.  Differences of 1.5 are exact."""
    from dosecuda_b200 import engine
    r80 = np.array([250.0], np.single)
    model = _model([4.0], [1.0], r80)
    model.lut_depths = model.lut_depths * np.float32(step)
    model.lut_idds = np.where(np.arange(400) % 2 == 0, np.float32(1.0), np.float32(3.0))[None].astype(np.single)
    grid = types.SimpleNamespace(spacing=np.array([2.0, 0.25, 2.0]), origin=np.array([0.0, -512.0, 0.0]))
    beam = types.SimpleNamespace(iso=np.zeros(3, np.single), gantry_angle=0.0, couch_angle=0.0,
                                 spot_list=np.array([[0.0, 0.0, 1.0, 0.0]], np.single))
    wet = np.random.default_rng(5).uniform(0.05, 24.9, (1, 4096, 1)).astype(np.single)
    dose = engine.proton_dose(torch.as_tensor(wet, device="cuda"), grid, beam, engine.ProtonModelDevice(model)).cpu().numpy()
    mm = (wet * np.float32(10.0)).astype(np.float64)
    idd = np.interp(mm, model.lut_depths[0].astype(np.float64), model.lut_idds[0].astype(np.float64))
    assert np.abs(dose / _influence64(wet, 250.0, 4.0, idd, 0.0) - 1.0).max() <= 1e-6
