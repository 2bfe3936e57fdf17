"""A photon beam's probe (dc_photon_beam_probe) under graph capture and on two streams at once."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_probe_captured_first_and_on_two_streams():
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTPlan

    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    shape, sp = (40, 44, 52), 3.0
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array([sp] * 3), origin=np.array([-n * sp / 2 for n in (nx, ny, nz)]))
    x12 = np.where(np.abs(model.mlc_offsets) <= 30.0, 25.0, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, 30.0, 0.0, 15.0, None, None)
    beam = engine.PhotonBeam(grid, shape)
    beam.set_density(torch.ones(shape, device="cuda"))
    beam.terma(model, cp)
    full = beam.dose().reshape(-1)
    n = full.numel()
    lists = [torch.arange(q, n, 7, device="cuda", dtype=torch.int32) for q in range(4)]
    outs = [torch.empty(v.numel(), device="cuda") for v in lists]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()  # the beam's first probe is the captured one
    with torch.cuda.graph(graph):
        beam.probe(lists[0], out=outs[0])
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(20):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for q, s in enumerate(streams):
            beam.probe(lists[q + 1], out=outs[q + 1], stream=s)
        graph.replay()
        torch.cuda.synchronize()
        for v, o in zip(lists, outs):
            assert torch.equal(o, full[v.long()])
