"""Photon beams (dc_photon_beam.cu) used from several threads and on several streams at once."""
import threading
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _beam(engine, model, shape, spacing, half_x, half_y=25.0, gantry=20.0):
    import torch

    from dosecuda_b200.plan_imrt import IMRTControlPoint
    nz, ny, nx = shape
    grid = types.SimpleNamespace(spacing=np.array([spacing] * 3),
                                 origin=np.array([-n * spacing / 2 for n in (nx, ny, nz)]))
    x12 = np.where(np.abs(model.mlc_offsets) <= half_y, half_x, 0.0)
    mlc = np.array(np.vstack((-x12, x12, model.mlc_offsets, model.mlc_widths)), dtype=np.single).T
    cp = IMRTControlPoint(np.zeros(3, np.single), 100.0, mlc, gantry, 0.0, 0.0, None, None)
    beam = engine.PhotonBeam(grid, shape)
    beam.set_density(torch.ones(shape, device="cuda"))
    return beam, cp


def test_doses_of_several_spacings_from_several_threads():
    """The CCCS of a fine grid opts in to more shared memory than that of a coarser one; either may run between
    the other's opt-in and its launch.  Every call has to be accepted and give the dose it gives alone."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    beams, want, outs = [], [], []
    for spacing in (1.0, 1.5, 1.25):
        beam, cp = _beam(engine, model, (8, 12, 16), spacing, 25.0)
        beam.terma(model, cp)
        beams.append(beam)
        want.append((beam.dose(), beam.probe()))
        outs.append((torch.empty_like(want[-1][0]), torch.empty_like(want[-1][1])))
    streams = [torch.cuda.Stream() for _ in beams]
    torch.cuda.synchronize()
    failed = []

    def work(q):
        try:
            for _ in range(400):
                beams[q].dose(out=outs[q][0], stream=streams[q])
                beams[q].probe(out=outs[q][1], stream=streams[q])
        except Exception as e:  # a launch that was refused
            failed.append(e)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(beams))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed[0]
    for (dose, probe), (d, p) in zip(want, outs):
        assert torch.equal(dose, d) and torch.equal(probe, p)


def test_termas_of_two_beams_on_two_streams():
    """Two beams' TERMA passes, enqueued on two streams without waiting and from two threads, share the
    context's head factors: each has to be what it is alone.  A photon dose call uses the same buffer."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    pairs = [_beam(engine, model, (48, 56, 64), 3.0, hx, hy, ga) for hx, hy, ga in ((60.0, 50.0, 0.0), (15.0, 30.0, 75.0))]
    want = [b.terma(model, cp, out=True).clone() for b, cp in pairs]
    torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    streams = [torch.cuda.Stream() for _ in pairs]
    for _ in range(10):
        got = []
        for (b, cp), s in zip(pairs, streams):
            with torch.cuda.stream(s):
                got.append(b.terma(model, cp, out=True, stream=s))
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g, w)
    bad = []

    def work(q):
        (b, cp), s = pairs[q], streams[q]
        with torch.cuda.stream(s):
            for _ in range(20):
                g = b.terma(model, cp, out=True, stream=s)
                s.synchronize()
                if not torch.equal(g, want[q]):
                    bad.append(q)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_kernels_timed_from_several_threads():
    """With the kernel profiler on, photon beams on several threads time their kernels while another thread reads
    the profile: every launch is counted once."""
    import torch

    from dosecuda_b200 import engine
    from dosecuda_b200.plan_imrt import IMRTPlan
    model = IMRTPlan("VarianTrueBeamHF").beam_models[0]
    beams = [_beam(engine, model, (8, 12, 16), 3.0, 25.0) for _ in range(3)]
    outs = [torch.empty((8, 12, 16), device="cuda") for _ in beams]
    streams = [torch.cuda.Stream() for _ in beams]
    for (b, cp), o in zip(beams, outs):
        b.terma(model, cp)
        b.dose(out=o)
    torch.cuda.synchronize()
    failed, n = [], 200

    def work(q):
        try:
            for _ in range(n):
                beams[q][0].dose(out=outs[q], stream=streams[q])
        except Exception as e:
            failed.append(e)

    engine.profile(0, enable=True, reset=True)
    try:
        threads = [threading.Thread(target=work, args=(q,)) for q in range(len(beams))]
        for t in threads:
            t.start()
        for _ in range(20):
            engine.profile(0)
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        counted = engine.profile(0)["cccs"][0]
    finally:
        engine.profile(0, enable=False)
    assert not failed, failed[0]
    assert counted == n * len(beams)
