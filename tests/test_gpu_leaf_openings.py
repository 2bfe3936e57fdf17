"""Collimator openings of the head transmission: closed leaf pairs left out, equal neighbours taken as one."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leaves(kind, model):
    """(x1, x2, offset, width) per pair in mm at the isocentre."""
    off, wid = np.array(model.mlc_offsets, np.float64), np.array(model.mlc_widths, np.float64)
    x1, x2 = np.where(np.abs(off) <= 30, -25.0, 0.0), np.where(np.abs(off) <= 30, 25.0, 0.0)
    if kind == "islands":      # open, closed in the middle of the opening (not at 0), open again
        mid = np.abs(off) <= 8
        x1, x2 = np.where(mid, 12.5, x1), np.where(mid, 12.5, x2)
    elif kind == "steps":      # two runs of equal pairs, then every pair another
        x2 = np.where((off > 0) & (x2 > 0), 31.0, x2)
        x1 = np.where(off > 15, x1 - 0.1 * off, x1)
    elif kind == "gap":        # equal pairs whose edges do not meet
        off = np.where(off > 2, off + 0.75, off)
    elif kind == "overlap":    # equal pairs that overlap
        wid = wid * 1.2
    elif kind == "descending":
        return np.stack((x1, x2, off, wid), 1)[::-1]
    return np.stack((x1, x2, off, wid), 1)


@pytest.mark.parametrize("kind", ["square", "islands", "steps", "gap", "overlap", "descending"])
def test_terma_equals_that_of_unmergeable_pairs(kind):
    """Against the same leaves with every second pair opened by one unit in the last place on its right side,
    so that no pair is closed and no two neighbours are equal.  That moves an edge by 2e-6 mm, 1e-6 of a
    source sigma; summing up to 20 pairs' erf differences by themselves adds 40 roundings of 6e-8 at most:
    5e-6 of the largest TERMA."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    shape, sp = (19, 22, 27), 5.0
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([-n * sp / 2 for n in (nx, ny, nz)]))
    beam = engine.PhotonBeam(grid, shape)
    beam.set_density(torch.ones(shape, device="cuda"))
    terma = []
    for apart in (False, True):
        mlc = np.ascontiguousarray(_leaves(kind, model), dtype=np.single)
        if apart:
            for q in range(len(mlc)):
                if mlc[q, 0] == mlc[q, 1] or q % 2:
                    mlc[q, 1] = np.nextafter(mlc[q, 1], np.single(100.0))
        cp = IMRTControlPoint(np.array([2.0, -1.0, 3.0], np.single), 100.0, mlc, 25.0, 35.0, 10.0, None, None)
        terma.append(beam.terma(model, cp, out=True).cpu().numpy())
    assert terma[0].max() > 0.1
    assert np.abs(terma[0] - terma[1]).max() <= 5e-6 * terma[0].max()


def test_leaf_edge_that_is_not_a_number():
    """A leaf pair at a y position of NaN makes TERMA NaN everywhere, also far beside the opening (here up to
    0.8 m), where the pair's x factor is exactly 0."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    x1, x2, off, wid = _leaves("square", model).T.copy()
    off[len(off) // 2] = np.nan
    shape = (3, 4, 200)
    grid = types.SimpleNamespace(spacing=np.array([8.0, 4.0, 4.0]), origin=np.array([-800.0, -8.0, -6.0]))
    mlc = np.array(np.vstack((x1, x2, off, wid)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, 0.0, 0.0, 0.0, None, None)
    beam = engine.PhotonBeam(grid, shape)
    beam.set_density(torch.ones(shape, device="cuda"))
    assert bool(beam.terma(model, cp, out=True).isnan().all())
