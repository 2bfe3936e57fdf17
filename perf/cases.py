"""The calls this framework is used for, with sizes, for timing and for comparing results.

Proton (double-Gaussian pencil beam) and photon (TERMA + collapsed-cone) dose through the public entry
points: the drop-in functions on numpy volumes, the device-resident engine on torch CUDA tensors, the
batched plans and the differentiable forms that a plan optimiser calls.  Inputs are seeded phantoms: water,
or a body with HU noise in air, with bone, lung and air inserts and a spherical target, spot weights that are
lognormal, apertures that follow the target's outline with leaf jitter.

``exact`` restates each result in float64 torch: trilinear sampling with exact weights, float32 only where a
rounded coordinate decides which sample is taken.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from dosecuda_b200 import dose_kernels, engine
from dosecuda_b200.plan import VolumeObject
from dosecuda_b200.plan_impt import IMPTBeam, IMPTDoseGrid, IMPTPlan
from dosecuda_b200.plan_imrt import IMRTControlPoint, IMRTDoseGrid, IMRTPlan

# HU -> relative stopping power / density points of the shipped machines (both tables are the same)
HU_TABLE = (np.array([-1000.0, -742.5, -92.11, 0.0, 24.0, 36.0, 76.33, 1369.0, 3096.0]),
            np.array([0.00113, 0.25771, 0.9617, 1.00653, 1.02058, 1.03049, 1.07187, 1.74967, 2.36825]))

_PROTON = {"spacing": "2.0,2.0,2.0", "gantry": 0.0, "couch": 0.0, "shifter": 0, "target": 25.0, "pitch": 5.0,
           "hu": False, "body": True}
_PHOTON = {"spacing": "2.5", "gantry": 0.0, "couch": 0.0, "collimator": 0.0, "machine": "VarianTrueBeamHF", "energy": 0,
           "field": 100.0, "field_y": 100.0, "shaped": False, "body": False}


def listed():
    return [
        # the drop-in calls of the reference's plan loop, numpy in and out: one proton beam (ray trace, then
        # spots, the WET copied in between as the loop does) and one photon control point
        dict(_PROTON, name="proton_host_96", kind="proton_host", shape="96,96,96", body=False),
        dict(_PHOTON, name="photon_host_128", kind="photon_host", shape="128,128,128"),
        # device-resident proton beams: a small QA phantom, an oblique beam with the range shifter on an odd
        # anisotropic grid, and a clinical-size CT
        dict(_PROTON, name="proton_beam_small", kind="proton_beam", shape="36,40,44", spacing="3.0,3.0,3.0", target=15.0),
        dict(_PROTON, name="proton_beam_oblique", kind="proton_beam", shape="91,113,127", spacing="2.0,2.0,2.5", gantry=235.0,
             couch=30.0, shifter=1, target=30.0, hu=True),
        dict(_PROTON, name="proton_beam_clinic", kind="proton_beam", shape="160,256,256", spacing="1.5,1.5,2.0",
             gantry=71.7, target=32.0, hu=True),
        # one dose iteration of several plans at new spot weights, WETs in hand
        dict(_PROTON, name="proton_batch", kind="proton_batch", shape="96,160,160", spacing="2.0,2.0,2.5", plans=3, beams=2,
             target=30.0),
        # forward and backward of a plan optimiser at the objective's voxels
        dict(_PROTON, name="proton_opt_list", kind="proton_opt", shape="112,160,160", spacing="1.5,1.5,2.0", gantry=310.0,
             target=35.0, pitch=4.5, list=True),
        # device-resident photon control points: a small QA field, the standard open field, and a shaped
        # field at oblique angles on an odd grid with a body in air
        dict(_PHOTON, name="photon_cp_small", kind="photon_cp", shape="30,32,36", spacing="4.0", field=40.0, field_y=50.0),
        dict(_PHOTON, name="photon_cp_128", kind="photon_cp", shape="128,128,128"),
        dict(_PHOTON, name="photon_cp_oblique", kind="photon_cp", shape="97,131,143", spacing="3.0", gantry=40.0, couch=10.0,
             collimator=15.0, machine="ElektaVersaSibAxesse", field=140.0, field_y=120.0, shaped=True, body=True),
        # a modulated arc as one plan call, from HU
        dict(_PHOTON, name="photon_arc", kind="photon_arc", shape="128,128,128", spacing="2.5", cps=12, shaped=True, body=True,
             field=90.0, field_y=90.0),
        # forward and adjoint of a beamlet-fluence optimiser
        dict(_PHOTON, name="photon_fluence", kind="photon_fluence", shape="64,72,80", spacing="3.0", gantry=25.0,
             field=80.0, field_y=70.0, body=True),
    ]


def _dims(rng, lo, hi):
    return [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["proton_host", "proton_beam", "proton_beam", "proton_batch", "proton_opt", "proton_opt",
                       "photon_host", "photon_cp", "photon_cp", "photon_arc", "photon_fluence"])
    if kind.startswith("proton"):
        c = dict(_PROTON, kind=kind)
        sp = rng.choice([1.5, 2.0, 2.5, 3.0])
        iso = kind == "proton_host"  # the drop-in loop takes isotropic grids only
        d = {"proton_host": _dims(rng, 40, 128), "proton_beam": _dims(rng, 36, 200), "proton_batch": _dims(rng, 60, 110),
             "proton_opt": _dims(rng, 60, 140)}[kind]
        c["shape"] = ",".join(map(str, d))
        c["spacing"] = "%g,%g,%g" % (sp, sp, sp if iso else rng.choice([sp, 2.0, 2.5]))
        c["gantry"] = rng.choice([0.0, 90.0, 180.0, 270.0, round(rng.uniform(0, 360), 1), round(rng.uniform(0, 360), 1)])
        c["couch"] = rng.choice([0.0, 0.0, round(rng.uniform(-45, 45), 1)])
        c["shifter"] = rng.choice([0, 0, 1])
        c["target"] = round(rng.uniform(0.12, 0.2) * sp * min(d), 1)
        c["pitch"] = round(rng.uniform(4.0, 6.0), 2)
        c["hu"] = kind == "proton_beam" and rng.random() < 0.5
        c["body"] = rng.random() < 0.8
        if kind == "proton_batch":
            c.update(plans=rng.randint(1, 3), beams=rng.randint(1, 2))
        if kind == "proton_opt":
            c["list"] = rng.random() < 0.6
        return c
    c = dict(_PHOTON, kind=kind)
    hi = {"photon_arc": 110, "photon_fluence": 80}.get(kind, 150)
    d = _dims(rng, 30, hi)
    sp = rng.choice([2.0, 2.5, 2.5, 3.0, 4.0])
    c["shape"], c["spacing"] = ",".join(map(str, d)), "%g" % sp
    c["gantry"] = rng.choice([0.0, 90.0, round(rng.uniform(0, 360), 1), round(rng.uniform(0, 360), 1)])
    c["couch"] = rng.choice([0.0, 0.0, round(rng.uniform(-30, 30), 1)])
    c["collimator"] = rng.choice([0.0, round(rng.uniform(0, 90), 1)])
    c["machine"], c["energy"] = rng.choice([("VarianTrueBeamHF", 0), ("VarianTrueBeamHF", 1), ("ElektaVersaSibAxesse", 0),
                                            ("ElektaVersaSibAxesse", 1)])
    most = min(200.0, 0.7 * sp * min(d))
    c["field"], c["field_y"] = round(rng.uniform(20.0, max(25.0, most)), 1), round(rng.uniform(20.0, max(25.0, most)), 1)
    c["shaped"], c["body"] = kind != "photon_fluence" and rng.random() < 0.5, rng.random() < 0.6
    if kind == "photon_arc":
        c["cps"] = rng.randint(3, 10)
    return c


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _proton_model(shifter):
    return IMPTPlan().beam_models[shifter]


@functools.lru_cache(maxsize=None)
def _proton_device_model(shifter):
    return engine.ProtonModelDevice(_proton_model(shifter))


@functools.lru_cache(maxsize=None)
def _photon_model(machine, energy):
    return IMRTPlan(machine).beam_models[energy]


def _shape(case):
    return tuple(int(v) for v in case["shape"].split(","))


def _spacing(case):
    v = [float(x) for x in case["spacing"].split(",")]
    return v * 3 if len(v) == 1 else v


def _rng(case, seed, more=0):
    return np.random.default_rng([seed, more])


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _hu(shape, spacing, seed, body, target, centre):
    """(nz, ny, nx) float32 HU on the GPU: plain water filling the grid or, with ``body``, an ellipsoidal body of
    noisy water (20 +- 40 HU) in air; one bone cylinder, one lung block, one air pocket, and a target sphere of
    plain tissue."""
    rng = _rng(None, seed, 1)
    dev = _dev()
    g = torch.Generator(device="cpu").manual_seed(int(seed) % (1 << 31))
    nz, ny, nx = shape
    ext = np.array([nx, ny, nz]) * np.array(spacing)
    ax = [((torch.arange(n, device=dev, dtype=torch.float32) + 0.5) * s - n * s / 2) for n, s in zip((nx, ny, nz), spacing)]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    noise = torch.randn((1 << 16,), generator=g).to(dev)
    at = (torch.arange(nx, device=dev)[None, None, :] * 7919 + torch.arange(ny, device=dev)[None, :, None] * 104729
          + torch.arange(nz, device=dev)[:, None, None] * 1299709)
    hu = 20.0 + 40.0 * noise[(at + (at >> 7)) & 0xffff] if body else torch.zeros(shape, device=dev)
    c = rng.uniform(-0.25, 0.25, 2) * ext[[0, 2]]
    hu[((X - float(c[0])) ** 2 + (Z - float(c[1])) ** 2 < 12.0 ** 2).expand(hu.shape)] = 1000.0
    c = rng.uniform(-0.3, 0.3, 3) * ext
    h = np.minimum(rng.uniform(20.0, 35.0, 3), ext / 5)
    hu[((X - float(c[0])).abs() < float(h[0])) & ((Y - float(c[1])).abs() < float(h[1])) & ((Z - float(c[2])).abs() < float(h[2]))] = -700.0
    c = rng.uniform(-0.3, 0.3, 3) * ext
    hu[(X - float(c[0])) ** 2 + (Y - float(c[1])) ** 2 + (Z - float(c[2])) ** 2 < 8.0 ** 2] = -1000.0
    hu[(X - float(centre[0])) ** 2 + (Y - float(centre[1])) ** 2 + (Z - float(centre[2])) ** 2 < target ** 2] = 30.0
    if body:
        a = 0.45 * ext
        hu[(X / float(a[0])) ** 2 + (Y / float(a[1])) ** 2 + (Z / float(a[2])) ** 2 > 1.0] = -1000.0
    return hu.contiguous()


def _table(hu):
    """np.interp(hu, *HU_TABLE) as float32, on the volume's device."""
    x = torch.as_tensor(HU_TABLE[0], device=hu.device)
    y = torch.as_tensor(HU_TABLE[1], device=hu.device)
    v = hu.double()
    i = torch.clamp(torch.searchsorted(x, v, right=True) - 1, 0, x.numel() - 2)
    return (y[i] + (y[i + 1] - y[i]) / (x[i + 1] - x[i]) * (v.clamp(float(x[0]), float(x[-1])) - x[i])).float()


def _grid(cls, shape, spacing):
    g = cls()
    g.origin = np.array([-n * s / 2.0 for n, s in zip(shape[::-1], spacing)])
    g.spacing = np.array(spacing)
    g.size = np.array(shape)
    return g


def _target_centre(case, seed):
    if case["kind"] == "proton_opt":  # the plan, and with it the number of voxels and spots, is the case's own
        seed = 0
    ext = np.array(_shape(case)[::-1]) * np.array(_spacing(case))
    return (_rng(case, seed, 2).uniform(-0.06, 0.06, 3) * ext).astype(np.float32)


def _proton_beam(case, seed, gantry, more=0):
    """Energy layers about 3 mm of range apart over the target, spots on a square grid over its outline."""
    rng = _rng(case, seed, 10 + more)
    iso = _target_centre(case, seed)
    r = case["target"]
    ext = np.array(_shape(case)[::-1]) * np.array(_spacing(case))
    a = np.deg2rad(gantry)
    toward = np.array([math.sin(a), -math.cos(a), 0.0])  # source direction in the image frame, couch aside
    half = 0.45 * ext if case["body"] else 0.5 * ext
    if case["body"]:  # distance from the target to the body's surface
        qa, qb, qc = ((toward / half) ** 2).sum(), 2 * (iso * toward / half ** 2).sum(), ((iso / half) ** 2).sum() - 1.0
        depth = (-qb + math.sqrt(max(qb * qb - 4 * qa * qc, 0.0))) / (2 * qa)
    else:
        depth = min((half[i] - math.copysign(1, toward[i]) * iso[i]) / abs(toward[i]) for i in (0, 1) if abs(toward[i]) > 1e-6)
    r80 = _proton_model(case["shifter"]).divergence_params[:, 1].astype(np.float64)
    first = 20 if case["shifter"] else 0
    ids = []
    for w in np.arange(depth - r, depth + r + 3.0, 3.0):
        e = first + int(np.argmin(np.abs(r80[first:] - w)))
        if e not in ids:
            ids.append(e)
    n = int(math.ceil((r + 5.0) / case["pitch"]))
    pos = np.arange(-n, n + 1) * case["pitch"]
    gx, gy = np.meshgrid(pos, pos)
    keep = gx ** 2 + gy ** 2 <= (r + 5.0) ** 2
    gx, gy = gx[keep], gy[keep]
    beam = IMPTBeam()
    beam.spot_list = np.vstack([np.column_stack((gx, gy, rng.lognormal(0.0, 0.5, gx.size), np.full(gx.size, e))) for e in ids]).astype(np.single)
    beam.n_spots = len(beam.spot_list)
    beam.gantry_angle, beam.couch_angle, beam.iso = float(gantry), float(case["couch"]), iso
    beam.dicom_rangeshifter_label = "4" if case["shifter"] else "0"
    return beam


def _control_point(case, seed, gantry, more=0):
    """Leaves set to the field's rectangle, or (shaped) to an ellipse of its size with jitter on every leaf."""
    model = _photon_model(case["machine"], case["energy"])
    rng = _rng(case, seed, 40 + more)
    off, wid = np.asarray(model.mlc_offsets, np.float64), np.asarray(model.mlc_widths, np.float64)
    fx, fy = case["field"] / 2, case["field_y"] / 2
    inside = np.abs(off) <= fy
    if not inside.any():
        inside = np.abs(off) <= np.abs(off).min()
    half = np.where(inside, fx, 0.0)
    if case["shaped"]:
        half = np.where(inside, fx * np.sqrt(np.clip(1.0 - (off / (fy + 3.0)) ** 2, 0.05, 1.0)), 0.0)
    jit = rng.uniform(-0.25, 0.25, (2, off.size)) * half if case["shaped"] else np.zeros((2, off.size))
    mlc = np.array(np.vstack((-half + jit[0], half + jit[1], off, wid)), dtype=np.single).T
    return IMRTControlPoint(_target_centre(case, seed), float(rng.uniform(50.0, 150.0)), mlc, float(gantry), float(case["collimator"]),
                            float(case["couch"]), None, None)


def _march(rho, case, beam, model):
    """A beam's WET (cm) as a program has it in hand: straight 2 mm steps towards the source."""
    geo = _Geometry(case, beam.iso, beam.gantry_angle, beam.couch_angle, 0.0, (model.VSADX + model.VSADY) / 2)
    nz, ny, nx = rho.shape
    p = geo.voxels(rho.device).float()
    u = geo.src.to(p) - p
    u = u / u.norm(dim=1, keepdim=True)
    sp, iso = geo.sp.to(p), geo.iso.to(p)
    size = torch.tensor([nx, ny, nz], device=p.device, dtype=p.dtype)
    wet = torch.zeros(p.shape[0], device=p.device)
    vol = rho.float().reshape(-1)
    for t in range(int(math.ceil(float((sp * size).norm()) / 2.0)) + 1):
        q = torch.round((p + u * (2.0 * t + 0.5) + iso) / sp)
        ok = ((q >= 0) & (q < size)).all(1)
        if not bool(ok.any()):
            break
        i = q.clamp(min=torch.zeros_like(size), max=size - 1).long()
        wet += torch.where(ok, vol[i[:, 0] + nx * (i[:, 1] + ny * i[:, 2])], torch.zeros_like(wet)) * 0.2
    return wet.reshape(rho.shape).contiguous()


def _objective_voxels(case, seed):
    """Flat indices of the target and of a ring of tissue beside it, ascending."""
    nz, ny, nx = _shape(case)
    c, r = _target_centre(case, seed), case["target"]
    sp = _spacing(case)
    ax = [((torch.arange(n, device=_dev(), dtype=torch.float32) + 0.5) * s - n * s / 2) for n, s in zip((nx, ny, nz), sp)]
    d2 = (ax[0][None, None, :] - float(c[0])) ** 2 + (ax[1][None, :, None] - float(c[1])) ** 2 + (ax[2][:, None, None] - float(c[2])) ** 2
    ring = (d2 > (r + 6.0) ** 2) & (d2 < (r + 10.0) ** 2) & (ax[1][None, :, None] > float(c[1]))
    return torch.nonzero(((d2 < r ** 2) | ring).reshape(-1)).reshape(-1).int()


def _object(grid, data):
    v = VolumeObject()
    v.voxel_data = np.array(data, dtype=np.single)
    v.origin = np.array(grid.origin, dtype=np.single)
    v.spacing = np.array(grid.spacing, dtype=np.single)
    return v


def _fluence(na, nb, seed):
    return torch.as_tensor(_rng(None, seed, 70).uniform(0.2, 1.8, (nb, na)).astype(np.float32), device=_dev())


def _smooth_noise(shape, seed, scale):
    g = torch.Generator(device="cpu").manual_seed((int(seed) + 77) % (1 << 31))
    n = torch.randn((1 << 15,), generator=g).to(_dev())
    i = torch.arange(int(np.prod(shape)), device=_dev())
    return (scale * n[(i * 48271 + (i >> 9)) & 0x7fff]).reshape(shape).contiguous()


def prepare(case, seed):
    shape, sp, kind = _shape(case), _spacing(case), case["kind"]
    hu = _hu(shape, sp, seed, case["body"], case.get("target", 20.0), _target_centre(case, seed))
    s = {"kind": kind}
    if kind.startswith("proton"):
        s["grid"] = _grid(IMPTDoseGrid, shape, sp)
        s["model"] = _proton_model(case["shifter"])
        s["beam"] = _proton_beam(case, seed, case["gantry"])
        rho = _table(hu)
        if kind == "proton_host":
            s["volume"] = _object(s["grid"], rho.cpu().numpy())
        elif kind == "proton_beam":
            s.update(volume=hu if case["hu"] else rho, hu=case["hu"], dmodel=_proton_device_model(case["shifter"]))
        elif kind == "proton_batch":
            b = s["batch"] = engine.ProtonBatch(s["model"])
            for p in range(case["plans"]):
                vol = rho if p == 0 else _table(_hu(shape, sp, seed + 1000 * p, case["body"], case["target"], _target_centre(case, seed)))
                pid = b.add_plan(s["grid"], vol)
                for q in range(case["beams"]):
                    b.add_beam(pid, _proton_beam(case, seed, _batch_gantry(case, p, q), more=1 + 5 * p + q))
            b.commit()
            beams = [_proton_beam(case, seed, _batch_gantry(case, p, q), more=1 + 5 * p + q) for p in range(case["plans"]) for q in range(case["beams"])]
            for i, bm in enumerate(beams):
                b.wets[i].copy_(_march(b.rlsp[b.beam_plan[i]], case, bm, s["model"]))
            s["mu"] = b.mu0 * torch.as_tensor(_rng(case, seed, 3).uniform(0.5, 1.5, b.n_spots).astype(np.float32), device=_dev())
        else:
            s["wet"] = _march(rho, case, s["beam"], s["model"])
            s["plan"] = engine.ProtonBeamPlan(s["grid"], s["beam"], s["model"])
            s["mu"] = s["plan"].mu.clone().requires_grad_(True)
            if case["list"]:
                s["voxels"] = _objective_voxels(case, seed)
                s["grad"] = _smooth_noise((s["voxels"].numel(),), seed, 1.0)
            else:
                s["grad"] = torch.zeros(shape, device=_dev())
                v = _objective_voxels(case, seed).long()
                s["grad"].reshape(-1)[v] = _smooth_noise((v.numel(),), seed, 1.0)
        return s
    s["grid"] = _grid(IMRTDoseGrid, shape, sp)
    s["model"] = _photon_model(case["machine"], case["energy"])
    if kind == "photon_arc":
        step = 360.0 / case["cps"]
        s.update(volume=hu, cps=[_control_point(case, seed, case["gantry"] + step * q, more=q) for q in range(case["cps"])])
        s["weights"] = [float(s["model"].outputFactor(cp)) for cp in s["cps"]]
        return s
    s["cp"] = _control_point(case, seed, case["gantry"])
    rho = _table(hu)
    if kind == "photon_host":
        s["volume"] = _object(s["grid"], rho.cpu().numpy())
    elif kind == "photon_cp":
        s["volume"] = rho
    else:
        s["beam"] = engine.PhotonFluenceBeam.field_map(rho, s["grid"], s["model"], s["cp"])
        s["fluence"] = _fluence(s["beam"].na, s["beam"].nb, seed)
        s["grad"] = _smooth_noise(shape, seed, 1.0) * (_smooth_noise(shape, seed + 1, 1.0) > 0.0)
    return s


def _batch_gantry(case, p, q):
    return (case["gantry"] + 61.0 * p + 360.0 / case["beams"] * q + 13.0) % 360.0


def run(s):
    kind = s["kind"]
    if kind == "proton_host":
        wet = dose_kernels.proton_raytrace_cuda(s["model"], s["volume"], s["beam"], 0)
        dose = dose_kernels.proton_spot_cuda(s["model"], s["volume"], _object(s["grid"], wet), s["beam"], 0)
        return {"wet": wet, "dose": dose}
    if kind == "proton_beam":
        if s["hu"]:
            wet = engine.proton_wet_hu(s["volume"], s["grid"], s["beam"], s["model"], HU_TABLE)
        else:
            wet = engine.proton_wet(s["volume"], s["grid"], s["beam"], s["model"])
        return {"wet": wet, "dose": engine.proton_dose(wet, s["grid"], s["beam"], s["dmodel"])}
    if kind == "proton_batch":
        return {"doses": list(s["batch"].dose(s["mu"]))}
    if kind == "proton_opt":
        if "voxels" in s:
            dose = engine.proton_dose_list_autograd(s["mu"], s["wet"], s["plan"], s["voxels"])
        else:
            dose = engine.proton_dose_autograd(s["mu"], s["wet"], s["plan"])
        (grad,) = torch.autograd.grad(dose, s["mu"], s["grad"])
        return {"dose": dose.detach(), "grad": grad}
    if kind == "photon_host":
        return {"dose": dose_kernels.photon_dose_cuda(s["model"], s["volume"], s["cp"], 0)}
    if kind == "photon_cp":
        return {"dose": engine.photon_dose(s["volume"], s["grid"], s["model"], s["cp"])}
    if kind == "photon_arc":
        total = torch.zeros(s["volume"].shape, dtype=torch.float32, device=s["volume"].device)
        engine.photon_plan_dose(s["volume"], s["grid"], s["model"], s["cps"], s["weights"], total, hu_table=HU_TABLE)
        return {"dose": total}
    return {"dose": s["beam"].dose(s["fluence"]), "grad": s["beam"].adjoint(s["grad"])}


# ---------------------------------------------------------------------------------------------------
# work: each input read once, each output written once; operations of the method's own sums
# ---------------------------------------------------------------------------------------------------
def work(case):
    kind, n, sp = case["kind"], int(np.prod(_shape(case))), _spacing(case)
    long = float(np.linalg.norm(np.array(_shape(case)[::-1]) * np.array(sp)))
    if kind.startswith("proton"):
        spots = len(_proton_beam(case, 0, case["gantry"]).spot_list)
        layers = max(1, int(2 * case["target"] / 3.0) + 2)
        per_layer = spots / layers
        pair = 22.0 + 2.0  # distance to the axis, two Gaussians, two sums
        near = min(1.0, (120.0 ** 2) / (4 * (case["target"] + 60.0) ** 2))
        dose = 0.35 * n * layers * per_layer * near * pair
        march = n * (0.3 * long) * 24.0 + n * 55 * 2.0
        if kind == "proton_batch":
            k = case["plans"] * case["beams"]
            return {"bytes": 4.0 * n * (k + case["plans"]) + 36.0 * spots * k, "flops": dose * k}
        if kind == "proton_opt":
            m = 4.5 * case["target"] ** 3 / (sp[0] * sp[1] * sp[2]) if case["list"] else n
            return {"bytes": 4.0 * m * (4 if case["list"] else 3) + 44.0 * spots, "flops": 2 * dose / 0.35 / n * m * 0.8}
        return {"bytes": 4.0 * n * (4 if kind == "proton_host" else 3) + 36.0 * spots, "flops": march + dose}
    kernel = _photon_model(case["machine"], case["energy"]).kernel
    samples = 12.0 * float(np.sum(np.floor(kernel[:, 5] / (sp[0] / 10.0)) + 1))
    ext = np.array(_shape(case)[::-1]) * np.array(sp)
    lit = n * min(1.0, (case["field"] + 20) * (case["field_y"] + 20) / float(ext[0] * ext[2]))
    one = lit * samples * 44.0 + n * 200.0
    times = {"photon_arc": case.get("cps", 1), "photon_fluence": 2}.get(kind, 1)
    return {"bytes": 8.0 * n * (2 if kind == "photon_fluence" else 1), "flops": one * times}


# ---------------------------------------------------------------------------------------------------
# float64
# ---------------------------------------------------------------------------------------------------
class _Geometry:
    """Voxel positions relative to the isocentre, source, and the image -> head rotation, in float64."""

    def __init__(self, case, iso, gantry, couch, collimator, sad):
        self.shape, self.sp = _shape(case), torch.tensor(_spacing(case), dtype=torch.float64)
        origin = np.array([-n * s / 2.0 for n, s in zip(self.shape[::-1], _spacing(case))], dtype=np.float32)
        self.iso = torch.tensor((np.asarray(iso, np.float32) - origin).astype(np.float64))
        g, t, c = (math.radians(v) for v in ((gantry + 180.0) % 360.0, couch, collimator))
        self.src = torch.tensor([-sad * math.sin(g) * math.cos(t), sad * math.cos(g), sad * math.sin(g) * math.sin(t)], dtype=torch.float64)

        def about_y(s, k):
            return torch.tensor([[k, 0, s], [0, 1, 0], [-s, 0, k]], dtype=torch.float64)

        rot = torch.tensor([[math.cos(g), math.sin(g), 0], [-math.sin(g), math.cos(g), 0], [0, 0, 1]], dtype=torch.float64)
        swap = torch.tensor([[-1, 0, 0], [0, 0, 1], [0, 1, 0]], dtype=torch.float64)
        self.to_head = swap @ about_y(-math.sin(c), math.cos(c)) @ rot @ about_y(-math.sin(t), math.cos(t))

    def voxels(self, dev):
        nz, ny, nx = self.shape
        k, j, i = torch.meshgrid(*(torch.arange(n, dtype=torch.float64, device=dev) for n in (nz, ny, nx)), indexing="ij")
        return torch.stack((i.reshape(-1), j.reshape(-1), k.reshape(-1)), 1) * self.sp.to(dev) - self.iso.to(dev)

    def texture(self, q):
        return (q + self.iso.to(q)) / self.sp.to(q) + 0.5


def _padded(vol, border):
    return torch.nn.functional.pad(vol.double(), (1, 2, 1, 2, 1, 2), value=border)


def _cells(tc, shape):
    """Flat index of the low corner in the padded volume, its eight offsets, and the eight weights."""
    nz, ny, nx = shape
    x = tc - 0.5
    hi = torch.tensor([nx, ny, nz], dtype=x.dtype, device=x.device)
    x = torch.minimum(x.clamp(min=-1.0), hi)
    f = torch.floor(x)
    a = x - f
    i = f.long() + 1
    row, plane = nx + 3, (nx + 3) * (ny + 3)
    base = i[:, 0] + row * i[:, 1] + plane * i[:, 2]
    out = []
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                w = (a[:, 0] if di else 1 - a[:, 0]) * (a[:, 1] if dj else 1 - a[:, 1]) * (a[:, 2] if dk else 1 - a[:, 2])
                out.append((base + di + row * dj + plane * dk, w))
    return out


def _wet64(rho, geo, border, smooth):
    """Radiological depth (cm): 1 mm samples until the texture coordinate leaves the volume."""
    dev = rho.device
    nz, ny, nx = geo.shape
    vol = _padded(rho, border).reshape(-1)
    p = geo.voxels(dev)
    u = geo.src.to(dev) - p
    u = u / u.norm(dim=1, keepdim=True)
    size = torch.tensor([nx, ny, nz], dtype=torch.float64, device=dev)
    wet = torch.full((p.shape[0],), -0.05, dtype=torch.float64, device=dev)
    live = torch.arange(p.shape[0], device=dev)
    t = 0
    while live.numel():
        tc = geo.texture(p + u * float(t))
        ok = ((tc.float() >= 0) & (tc.float() < size.float())).all(1)
        if not bool(ok.all()):
            live, p, u, tc = live[ok], p[ok], u[ok], tc[ok]
        if not live.numel():
            break
        r = sum(vol[i] * w for i, w in _cells(tc, geo.shape))
        wet[live] += 0.1 * r.clamp(min=0.0)
        t += 1
    if not smooth:
        return wet
    p32 = geo.voxels(dev).float()
    r32 = geo.to_head.to(dev).float()
    iso, sp = geo.iso.to(dev).float(), geo.sp.to(dev).float()
    h = p32 @ r32.T
    total, count, reach = wet.clone(), torch.ones_like(wet), wet.float() * 10.0
    for d in range(6):
        ang = np.float32(d) * np.float32(math.pi) / np.float32(3.0)
        s, c = float(np.float32(math.sin(ang))), float(np.float32(math.cos(ang)))
        for dr in range(1, 10):
            q = torch.stack((h[:, 0] + dr * c, h[:, 1] + dr * s, h[:, 2]), 1) @ r32
            v = (q + iso) / sp
            i = (torch.sign(v) * torch.floor(v.abs() + 0.5)).long()
            ok = ((i >= 0) & (i < size.long())).all(1) & (float(dr) < reach)
            j = (i[:, 0] + nx * (i[:, 1] + ny * i[:, 2])).clamp(0, wet.numel() - 1)
            total += torch.where(ok, wet[j], torch.zeros_like(wet))
            count += ok
    return total / count


def _pencil64(wet, geo, beam, model, mu=None, voxels=None, grad=None):
    """Dose (flat) of the beam; with ``grad`` also each spot's sum of grad x dose per MU."""
    dev = wet.device
    p = geo.voxels(dev)
    w = wet.reshape(-1).float().mul(10.0).double()
    if voxels is not None:
        p, w = p[voxels.long()], w[voxels.long()]
    h = p @ geo.to_head.to(dev).T
    dist = (geo.src.to(dev) - p).norm(dim=1)
    spots = torch.as_tensor(np.asarray(beam.spot_list, np.float64), device=dev)
    weight = spots[:, 2] if mu is None else mu.detach().double()
    dose = torch.zeros(w.shape[0], dtype=torch.float64, device=dev)
    back = torch.zeros(spots.shape[0], dtype=torch.float64, device=dev)
    dvp = np.asarray(model.divergence_params, np.float64)
    for e in np.unique(np.asarray(beam.spot_list)[:, 3]).astype(int):
        r80, A, B, C = (float(v) for v in dvp[e, 1:5])
        inside = torch.nonzero(~(w.float() > np.float32(1.1) * np.float32(r80))).reshape(-1)
        which = torch.nonzero(spots[:, 3].long() == int(e)).reshape(-1)
        if not inside.numel():
            continue
        D, S, I = (torch.as_tensor(np.asarray(t[e], np.float64), device=dev) for t in (model.lut_depths, model.lut_sigmas, model.lut_idds))
        x = w[inside]
        q = torch.searchsorted(D, x)
        lo, hi = (q - 1).clamp(min=0), q.clamp(max=D.numel() - 1)
        f = torch.where(hi > lo, (x - D[lo]) / (D[hi] - D[lo]).clamp(min=1e-30), torch.zeros_like(x))
        idd, sig = I[lo] + (I[hi] - I[lo]) * f, S[lo] + (S[hi] - S[lo]) * f
        d = dist[inside] - x + 0.7 * r80
        st = (A * d + B) * d + C + sig
        c = torch.minimum(x.clamp(min=0.1), torch.full_like(x, r80 - 0.1))
        hs = 2.85 + 0.0014 * r80 * torch.log(c + 3.0) + 0.06 * c - 7.4e-5 * c * c - 0.22 * r80 / (c - r80 - 5.0) ** 2
        hw = (0.052 * torch.log(1.13 + c / (11.2 - 0.023 * r80)) + 0.35 * (0.0017 * r80 * r80 - r80) / ((r80 + 3.0) ** 2 - c * c)
              - 1.61e-9 * c * (r80 + 3.0) ** 2)
        sht = torch.sqrt(st * st + hs.clamp(min=0.0) ** 2)
        hw = hw.clamp(0.0, 0.9)
        pf, hf = (1 - hw) * idd / (2 * math.pi * st * st), hw * idd / (2 * math.pi * sht * sht)
        s = spots[which]
        tx, ty = s[:, 0] / model.VSADX, s[:, 1] / model.VSADY
        t2 = tx * tx + ty * ty + 1.0
        step = max(1, 8_000_000 // max(1, which.numel()))
        for a in range(0, inside.numel(), step):
            z = slice(a, min(inside.numel(), a + step))
            hv = h[inside[z]]
            rx, ry, rz = hv[:, 0:1] - s[None, :, 0], hv[:, 1:2] - s[None, :, 1], hv[:, 2:3]
            r2 = ((ry + rz * ty) ** 2 + (rx + rz * tx) ** 2 + (rx * ty - ry * tx) ** 2) / t2
            k = pf[z, None] * torch.exp(r2 * (-0.5 / st[z] ** 2)[:, None]) + hf[z, None] * torch.exp(r2 * (-0.5 / sht[z] ** 2)[:, None])
            dose[inside[z]] += k @ weight[which]
            if grad is not None:
                back[which] += grad.reshape(-1)[inside[z]].double() @ k
    return (dose, back) if grad is not None else dose


def _head64(model, cp, h, distance, sigma):
    mlc = np.asarray(cp.mlc, np.float32).astype(np.float64)
    scale = (model.primary_source_distance - model.mlc_distance) / model.primary_source_distance
    div = (distance - h[:, 2]) / (model.mlc_distance - h[:, 2])
    k = 1.0 / (sigma * math.sqrt(2.0))
    out = torch.zeros_like(div)

    def edge(y, at):
        return torch.erf(((y * scale - at) * div + at) * k)

    for x1, x2, off, wid in mlc:
        if x1 != x2:
            out += 0.25 * (edge(x2, h[:, 0]) - edge(x1, h[:, 0])) * (edge(off + 0.5 * wid, h[:, 1]) - edge(off - 0.5 * wid, h[:, 1]))
    return out


def _terma64(rho, geo, model, cp):
    """(TERMA, electron term) of every voxel."""
    m, dev = model, rho.device
    wet = _wet64(rho, geo, 0.0012, False)
    h = geo.voxels(dev) @ geo.to_head.to(dev).T
    rc = torch.hypot(h[:, 0], h[:, 1]) * (m.primary_source_distance - h[:, 2]) / m.primary_source_distance
    pr, pi, ps = (torch.as_tensor(np.asarray(v, np.float64), device=dev) for v in (m.profile_radius, m.profile_intensities, m.profile_softening))
    q = torch.searchsorted(pr, rc)
    lo, hi = (q - 1).clamp(min=0), q.clamp(max=pr.numel() - 1)
    f = torch.where(hi > lo, (rc - pr[lo]) / (pr[hi] - pr[lo]).clamp(min=1e-30), torch.zeros_like(rc))
    oaf, soft = pi[lo] + (pi[hi] - pi[lo]) * f, ps[lo] + (ps[hi] - ps[lo]) * f
    tp = _head64(m, cp, h, m.primary_source_distance, m.primary_source_size)
    ts = _head64(m, cp, h, m.scatter_source_distance, m.scatter_source_size)
    ratio = ts / tp
    ratio = torch.where(ratio < 1.0, ratio, torch.ones_like(ratio))
    total = torch.zeros_like(wet)
    gp = (m.primary_source_distance / (m.primary_source_distance - h[:, 2])) ** 2
    gs = m.scatter_source_distance / (m.scatter_source_distance - h[:, 2])
    for mu, pw, sw in zip(*(np.asarray(v, np.float64) for v in (m.spectrum_attenuation_coefficients, m.spectrum_primary_weights, m.spectrum_scatter_weights))):
        att = torch.exp(-mu * wet * soft)
        total += (1 - ratio) * pw * att * gp + ratio * sw * att * gs
    end = math.exp(-m.electron_attenuation * m.electron_fitted_dmax)
    el = ((torch.exp(-m.electron_attenuation * wet) - end) / (1 - end)).clamp(min=0.0)
    T = oaf * ((1 - m.scatter_source_weight) * tp * total + m.scatter_source_weight * ts * total)
    return T, m.electron_source_weight * (0.4 + 0.3 * ratio) * el * tp


def _cone64(rho, geo, model, mask, each):
    """Walks every cone direction of the voxels in ``mask`` outwards and hands ``each`` the sample's cells and
    its weight in the voxel's collapsed-cone sum (which is linear in the TERMA)."""
    dev = rho.device
    sp = float(np.float32(float(geo.sp[0])) / np.float32(10.0))
    rv = _padded(rho, 0.0012).reshape(-1)
    p = geo.voxels(dev)[mask]
    u = geo.src.to(dev) - p
    u = u / u.norm(dim=1, keepdim=True)
    axis = (geo.src / geo.src.norm()).to(dev)
    cosine = u @ axis
    ax = torch.linalg.cross(axis.expand_as(u), u)
    for theta, Am, am, Bm, bm, length in np.asarray(model.kernel, np.float32).astype(np.float64):
        at, left = [], np.float32(length)
        while left >= 0:
            at.append(float(np.float32(left * np.float32(10.0))))
            left = np.float32(left - np.float32(sp))
        for a in range(12):
            th, ph = math.radians(theta), a * math.pi / 6
            v = geo.to_head.T.to(dev) @ torch.tensor([math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)], dtype=torch.float64, device=dev)
            r = torch.linalg.cross(ax, v.expand_as(ax)) + cosine[:, None] * v + ax * ((ax @ v) / (1 + cosine))[:, None]
            far_p, far_s = torch.ones_like(cosine), torch.ones_like(cosine)
            for L in reversed(at):  # from the voxel outwards: everything nearer attenuates
                cells = _cells(geo.texture(p + r * L), geo.shape)
                D = sum(rv[i] * w for i, w in cells).clamp(min=float(np.float32(0.0012))) * sp
                e = torch.exp(-am * D)
                each(cells, math.sin(th) * (Am / am * (1 - e) * far_p + Bm * D * far_s))
                far_p, far_s = far_p * e, far_s * (1 - bm * D)


def _photon64(rho, case, model, cp, scale_terma=None):
    geo = _Geometry(case, cp.iso, cp.ga, cp.ta, cp.ca, model.primary_source_distance)
    T, el = _terma64(rho, geo, model, cp)
    mask = torch.nonzero(~(T.float() <= 0.01)).reshape(-1)
    scale = torch.ones_like(T) if scale_terma is None else scale_terma(geo)
    tv = _padded((T * scale).float().reshape(geo.shape), 0.0).reshape(-1)
    total = (el * scale)[mask].clone()

    def add(cells, w):
        total.add_(w * sum(tv[i] * c for i, c in cells))

    _cone64(rho, geo, model, mask, add)
    out = torch.zeros_like(T)
    out[mask] = total.clamp(min=0.0) * float(np.float32(np.float32(model.mu_calibration) * np.float32(cp.mu)))
    return out.reshape(geo.shape), T, el, mask, geo


def _fluence64(case, seed, rho, model, cp):
    mlc = np.asarray(cp.mlc, np.float32)
    openp = mlc[:, 1] > mlc[:, 0]
    pitch, margin = 5.0, 10.0
    a0, a1 = float(mlc[openp, 0].min()) - margin, float(mlc[openp, 1].max()) + margin
    b0, b1 = float((mlc[openp, 2] - 0.5 * mlc[openp, 3]).min()) - margin, float((mlc[openp, 2] + 0.5 * mlc[openp, 3]).max()) + margin
    na, nb = int(math.ceil((a1 - a0) / pitch)) + 1, int(math.ceil((b1 - b0) / pitch)) + 1
    F = _fluence(na, nb, seed).double().reshape(-1)
    kept = {}

    def modulate(geo):
        h = geo.voxels(rho.device) @ geo.to_head.to(rho.device).T
        sad = model.primary_source_distance
        fa = ((h[:, 0] * sad / (sad - h[:, 2]) - a0) / pitch).clamp(0.0, na - 1.0)
        fb = ((h[:, 1] * sad / (sad - h[:, 2]) - b0) / pitch).clamp(0.0, nb - 1.0)
        ia, ib = fa.floor().clamp(max=max(na - 2, 0)), fb.floor().clamp(max=max(nb - 2, 0))
        wa, wb = fa - ia, fb - ib
        i = ia.long() + na * ib.long()
        right, up = min(1, na - 1), na * min(1, nb - 1)
        kept["parts"] = [(i, (1 - wa) * (1 - wb)), (i + right, wa * (1 - wb)), (i + up, (1 - wa) * wb), (i + right + up, wa * wb)]
        return sum(F[j] * w for j, w in kept["parts"])

    dose, T, el, mask, geo = _photon64(rho, case, model, cp, modulate)
    shape = _shape(case)
    g = (_smooth_noise(shape, seed, 1.0) * (_smooth_noise(shape, seed + 1, 1.0) > 0.0)).double().reshape(-1)
    scale = float(np.float32(np.float32(model.mu_calibration) * np.float32(cp.mu)))
    back = torch.zeros((shape[0] + 3) * (shape[1] + 3) * (shape[2] + 3), dtype=torch.float64, device=rho.device)
    gm = g[mask] * scale

    def spread(cells, w):
        for i, c in cells:
            back.index_add_(0, i, gm * w * c)

    _cone64(rho, geo, model, mask, spread)
    inner = back.reshape(shape[0] + 3, shape[1] + 3, shape[2] + 3)[1:-2, 1:-2, 1:-2].reshape(-1)
    per_voxel = T * inner
    per_voxel[mask] += el[mask] * gm
    out = torch.zeros(na * nb, dtype=torch.float64, device=rho.device)
    for j, w in kept["parts"]:
        out.index_add_(0, j, per_voxel * w)
    return {"dose": dose, "grad": out.reshape(nb, na)}


@torch.no_grad()
def exact(case, seed):
    shape, sp, kind = _shape(case), _spacing(case), case["kind"]
    if not torch.cuda.is_available():
        return None  # minutes on a CPU
    hu = _hu(shape, sp, seed, case["body"], case.get("target", 20.0), _target_centre(case, seed))
    rho = _table(hu)
    if kind.startswith("proton"):
        model = _proton_model(case["shifter"])

        def geometry(b):
            return _Geometry(case, b.iso, b.gantry_angle, b.couch_angle, 0.0, (model.VSADX + model.VSADY) / 2)

        beam = _proton_beam(case, seed, case["gantry"])
        if kind in ("proton_host", "proton_beam"):
            geo = geometry(beam)
            wet = _wet64(rho, geo, 0.0, True)
            if rho.numel() * len(beam.spot_list) > 2e10:
                return {"wet": wet.reshape(shape), "dose": None}
            return {"wet": wet.reshape(shape), "dose": _pencil64(wet, geo, beam, model).reshape(shape)}
        if kind == "proton_batch":
            mu, at, doses = None, 0, []
            beams = [[_proton_beam(case, seed, _batch_gantry(case, p, q), more=1 + 5 * p + q) for q in range(case["beams"])] for p in range(case["plans"])]
            spots = sum(len(b.spot_list) for bs in beams for b in bs)
            if rho.numel() * spots > 6e10:
                return None
            mu = torch.as_tensor(np.concatenate([b.spot_list[:, 2] for bs in beams for b in bs]), device=rho.device)
            mu = mu * torch.as_tensor(_rng(case, seed, 3).uniform(0.5, 1.5, spots).astype(np.float32), device=rho.device)
            for p, bs in enumerate(beams):
                vol = rho if p == 0 else _table(_hu(shape, sp, seed + 1000 * p, case["body"], case["target"], _target_centre(case, seed)))
                total = torch.zeros(rho.numel(), dtype=torch.float64, device=rho.device)
                for b in bs:
                    n = len(b.spot_list)
                    total += _pencil64(_march(vol, case, b, model), geometry(b), b, model, mu=mu[at:at + n])
                    at += n
                doses.append(total.reshape(shape))
            return {"doses": doses}
        wet = _march(rho, case, beam, model)
        v = _objective_voxels(case, seed)
        g = _smooth_noise((v.numel(),), seed, 1.0)
        if case["list"]:
            dose, grad = _pencil64(wet, geometry(beam), beam, model, voxels=v, grad=g)
            return {"dose": dose, "grad": grad}
        full = torch.zeros(rho.numel(), dtype=torch.float32, device=rho.device)
        full[v.long()] = g
        dose, grad = _pencil64(wet, geometry(beam), beam, model, grad=full)
        return {"dose": dose.reshape(shape), "grad": grad}
    model = _photon_model(case["machine"], case["energy"])
    if kind == "photon_arc":
        step, total = 360.0 / case["cps"], torch.zeros(shape, dtype=torch.float64, device=rho.device)
        for q in range(case["cps"]):
            cp = _control_point(case, seed, case["gantry"] + step * q, more=q)
            total += float(model.outputFactor(cp)) * _photon64(rho, case, model, cp)[0]
        return {"dose": total}
    cp = _control_point(case, seed, case["gantry"])
    if kind == "photon_fluence":
        return _fluence64(case, seed, rho, model, cp)
    return {"dose": _photon64(rho, case, model, cp)[0]}
