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
