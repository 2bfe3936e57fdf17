"""Radiological depth of small volumes: a ray's samples over eight lanes (dc_common.cuh march_lanes)."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing,gantry", [
    ((1, 1, 1), (3.0, 3.0, 3.0), 0.0),       # one ray, shorter than its lanes
    ((3, 5, 17), (2.0, 2.5, 3.0), 40.0),     # one voxel past a block's 16
    ((20, 16, 15), (1.0, 1.0, 1.0), 90.0),   # one short of it; rays about a batch of 16 samples long
    ((12, 70, 33), (2.0, 2.0, 2.0), 200.0),  # several batches
])
def test_terma_of_marched_depth(shape, spacing, gantry):
    """TERMA against the CPU oracle, which sums each ray by itself.  The oracle's sample weights are
    products of rounded fractions, the texture unit's are rounded products (1/512 of the density step
    of 0.2 at most): over up to 140 samples of 0.1 cm below 6e-3 cm in a straight sum and, their signs
    alternating, a tenth of that; times 0.3 per cm of attenuation 2e-4.  A sample lost or taken twice
    is 0.08 cm and moves TERMA by more than 3e-3."""
    import torch

    import oracle
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array(spacing), origin=np.array([-n * s / 2 for n, s in zip((nx, ny, nz), spacing)]))
    rho = np.random.default_rng(7).uniform(0.8, 1.0, shape).astype(np.single)
    x12 = np.where(np.abs(model.mlc_offsets) <= 80.0, 70.0, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.array([0.7, -1.1, 0.4], np.single), 100.0, mlc, gantry, 0.0, 0.0, None, None)
    was = engine.photon_depth_mode(0)
    engine.photon_depth_mode(0, "march")
    try:
        beam = engine.PhotonBeam(grid, shape)
        beam.set_density(torch.as_tensor(rho, device="cuda"))
        terma = beam.terma(model, cp, out=True).cpu().numpy()
    finally:
        engine.photon_depth_mode(0, was)
    ref = oracle.photon_dose(rho, spacing, grid.origin, model, cp.iso, cp.mu, cp.ga, cp.ca, cp.ta,
                             np.ascontiguousarray(cp.mlc), tex_mode=1, intermediates=True)[1]
    assert ref.max() > 0.1
    np.testing.assert_allclose(terma, ref, rtol=1e-3, atol=1e-6)
