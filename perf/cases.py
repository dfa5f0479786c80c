"""Performance cases: the calls a program that reconstructs or models PET data
makes through this package's public entry points, over the sizes it makes
them at.

A case is a dict of plain values.  `listed()` names the cases that are
measured by default and `draw(rng)` gives more of the same ranges;
`prepare(case, seed)` makes a program's inputs and the objects it keeps,
`run(state)` is one pass, `work(case)` the bytes and operations a pass cannot
do without, `tolerance(case)` how far another correct implementation may be,
and `exact(case, seed)` the values in 64-bit arithmetic, computed here in
plain torch.

Families (`case["family"]`):
  project     A x and A^T y over list-mode events (OperatorProjectorDevice)
  nll         Poisson log-likelihood and its gradient (autograd)
  osem        list-mode reconstruction (OSEM_GPU): Siddon with and without
              TOF, one ray or several, frames with motion, image-space PSF
  histo_osem  histogram reconstruction, distance-driven with projection PSF
  histo_op    A x and A^T y over one subset of a histogram
  sens        sensitivity images
  image_psf   image-space PSF and its adjoint (spatially variant or not)
  lrem        low-rank dynamic reconstruction
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(
    os.path.abspath(__file__))), "yrt-pet_b200"))

import pyyrtpet_b200 as yrt  # noqa: E402
from pyyrtpet_b200 import _lib as L  # noqa: E402
from pyyrtpet_b200 import synthetic  # noqa: E402
from pyyrtpet_b200.autograd import poisson_nll_fused  # noqa: E402

TOF_FWHM_PS = 214.0
TOF_NSTD = 5
EPS_FLT = 1.19209e-07
DENOM_THRESHOLD = 1e-35

# Scanners: axial FOV, crystal z, crystal transverse, depth, radius, crystals
# per ring, rings, DOI layers, ring difference, angle difference, block.
SCANNERS = {
    "small": (64, 4, 4, 10, 300, 256, 16, 1, 15, 2, 1),
    "preclinical": (48, 4, 4, 10, 90, 128, 12, 1, 11, 3, 1),
    "large": (256, 3.2, 3.2, 20, 410, 672, 80, 1, 79, 2, 1),
}


# -------------------------------------------------------------------- cases --
def listed():
    return [
        # The smallest calls: a few thousand events on a small grid (a data
        # set's first look, a unit of an iterative solver's inner loop).
        {"name": "project small", "family": "project", "scanner": "small",
         "nx": 32, "ny": 32, "nz": 16, "voxel": 4.0, "events": 4099,
         "subsets": 1, "projector": "S", "tof": True, "comp": False},
        # Training a network through the projector: loss and gradient of one
        # phantom's events, a grid whose sizes are not multiples of anything.
        {"name": "nll gradient tof", "family": "nll", "scanner": "small",
         "nx": 125, "ny": 127, "nz": 61, "voxel": 2.0, "events": 3000017,
         "tof": True, "comp": True},
        # A reconstruction with every setting at its default.
        {"name": "osem plain", "family": "osem", "scanner": "small",
         "nx": 128, "ny": 128, "nz": 64, "voxel": 2.0, "events": 1000000,
         "iterations": 2, "subsets": 5, "tof": False, "comp": False,
         "rays": 1, "frames": 1, "motion": False, "psf": "none",
         "corrections": False},
        # The large one: TOF with attenuation and randoms, clinical scanner.
        {"name": "osem tof large", "family": "osem", "scanner": "large",
         "nx": 256, "ny": 256, "nz": 160, "voxel": 2.0, "events": 20000000,
         "iterations": 3, "subsets": 10, "tof": True, "comp": True,
         "rays": 1, "frames": 1, "motion": False, "psf": "none",
         "corrections": True},
        # Several rays per crystal pair, default precision.
        {"name": "osem multi-ray", "family": "osem", "scanner": "large",
         "nx": 200, "ny": 200, "nz": 125, "voxel": 2.5, "events": 2000003,
         "iterations": 1, "subsets": 4, "tof": True, "comp": False,
         "rays": 4, "frames": 1, "motion": False, "psf": "none",
         "corrections": False},
        # Dynamic frames of uneven size with rigid motion per frame.
        {"name": "osem dynamic motion", "family": "osem", "scanner": "large",
         "nx": 128, "ny": 128, "nz": 80, "voxel": 4.0, "events": 6000000,
         "iterations": 1, "subsets": 10, "tof": True, "comp": True,
         "rays": 1, "frames": 12, "motion": True, "psf": "none",
         "corrections": False},
        # Resolution modelling in image space inside the reconstruction.
        {"name": "osem image psf", "family": "osem", "scanner": "large",
         "nx": 192, "ny": 192, "nz": 96, "voxel": 2.0, "events": 2000000,
         "iterations": 1, "subsets": 8, "tof": True, "comp": True,
         "rays": 1, "frames": 1, "motion": False, "psf": "uniform",
         "corrections": False},
        # Histogram reconstruction, distance-driven with projection PSF.
        {"name": "histogram dd psf", "family": "histo_osem",
         "scanner": "small", "nx": 200, "ny": 200, "nz": 100, "voxel": 2.5,
         "events": 20000000, "iterations": 1, "subsets": 12, "comp": True},
        # Forward and back projection of one subset of a histogram.
        {"name": "histogram operator", "family": "histo_op",
         "scanner": "small", "nx": 128, "ny": 128, "nz": 64, "voxel": 2.0,
         "subsets": 12, "projector": "S", "comp": False},
        # Sensitivity image of a scanner with an attenuation map.
        {"name": "sensitivity attenuated", "family": "sens",
         "scanner": "small", "nx": 128, "ny": 128, "nz": 64, "voxel": 2.0,
         "projector": "S", "comp": True, "mu": True},
        # Spatially variant PSF and its adjoint on one image.
        {"name": "variant psf", "family": "image_psf", "nx": 192, "ny": 192,
         "nz": 96, "voxel": 2.0, "frames": 1, "variant": True},
        # Low-rank dynamic reconstruction, temporal basis update.
        {"name": "low-rank dynamic", "family": "lrem", "scanner": "small",
         "nx": 128, "ny": 128, "nz": 64, "voxel": 2.0, "events": 2000000,
         "iterations": 1, "subsets": 4, "rank": 6, "frames": 20,
         "update_h": True, "comp": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, field, voxels, nz_field, scale=1.0):
    """A grid over about field mm: nx and ny between the voxel limits, equal
    or not, multiples of 4 or not."""
    voxel = rng.choice((1.5, 2.0, 2.5, 3.0, 4.0)) * scale
    nx = min(voxels[1], max(voxels[0], int(round(field * rng.uniform(0.7, 1.1) / voxel))))
    ny = nx if rng.random() < 0.5 else min(voxels[1], max(voxels[0], nx + rng.randint(-9, 9)))
    nz = max(4, int(round(nz_field * rng.uniform(0.7, 1.0) / voxel)))
    if rng.random() < 0.5:
        nx, ny, nz = nx - nx % 4 or 4, ny - ny % 4 or 4, nz - nz % 2 or 2
    return {"nx": nx, "ny": ny, "nz": nz, "voxel": voxel}


def draw(rng):
    family = rng.choice(("project", "nll", "osem", "osem", "osem", "histo_osem",
                         "histo_op", "sens", "image_psf", "lrem"))
    case = {"family": family}
    if family == "image_psf":
        case.update(_grid(rng, 400, (24, 256), 250))
        case.update(frames=rng.choice((1, 1, 2, 3)), variant=rng.random() < 0.5)
        return case
    if family in ("histo_osem", "histo_op", "sens"):
        case["scanner"] = rng.choice(("small", "preclinical"))
    else:
        case["scanner"] = rng.choice(("small", "preclinical", "large"))
    field = {"small": 260, "preclinical": 110, "large": 500}[case["scanner"]]
    depth = SCANNERS[case["scanner"]][0]
    case.update(_grid(rng, field, (24, 250), depth,
                      0.5 if case["scanner"] == "preclinical" else 1.0))
    case["comp"] = rng.random() < 0.5
    if family == "project":
        case.update(events=_log_int(rng, 2000, 4000000), subsets=rng.choice((1, 1, 3, 8)),
                    projector=rng.choice(("S", "S", "S", "DD")), tof=rng.random() < 0.6)
    elif family == "nll":
        case.update(events=_log_int(rng, 20000, 4000000), tof=rng.random() < 0.7)
    elif family == "osem":
        kind = rng.choice(("one", "one", "rays", "frames", "psf"))
        case.update(events=_log_int(rng, 50000, 5000000), iterations=rng.choice((1, 2, 3)),
                    subsets=rng.choice((1, 4, 5, 10)), tof=rng.random() < 0.6,
                    rays=rng.choice((2, 3, 4)) if kind == "rays" else 1,
                    frames=rng.choice((4, 8, 12)) if kind == "frames" else 1,
                    motion=kind == "frames" and rng.random() < 0.6,
                    psf=rng.choice(("uniform", "variant")) if kind == "psf" else "none",
                    corrections=rng.random() < 0.5)
        if kind == "rays":
            case["events"] = min(case["events"], 2000000)
    elif family == "histo_osem":
        case.update(events=_log_int(rng, 500000, 20000000), iterations=1,
                    subsets=rng.choice((4, 12)))
    elif family == "histo_op":
        case.update(subsets=rng.choice((6, 12, 24)), projector=rng.choice(("S", "S", "DD")))
    elif family == "sens":
        case.update(projector=rng.choice(("S", "S", "DD")), mu=rng.random() < 0.5)
    else:
        case.update(events=_log_int(rng, 100000, 2000000), iterations=1,
                    subsets=rng.choice((2, 4)), rank=rng.randint(2, 10),
                    frames=rng.randint(6, 24), update_h=rng.random() < 0.5)
        case["scanner"] = "small"
        case.update(_grid(rng, 260, (24, 128), 64))
    return case


# ------------------------------------------------------------------- inputs --
def _scanner(case):
    return yrt.Scanner(case["scanner"], *SCANNERS[case["scanner"]])


def _image_params(case, frames=1):
    v = case["voxel"]
    return yrt.ImageParams(case["nx"], case["ny"], case["nz"], case["nx"] * v,
                           case["ny"] * v, case["nz"] * v, nt=frames)


def _phantom(case, seed):
    """A cylinder with spheres that fits the scanner and the grid."""
    axial, radius = SCANNERS[case["scanner"]][0], SCANNERS[case["scanner"]][4]
    ph = synthetic.random_phantom(seed, axial / 2)
    k = min(1.0, 0.45 * min(case["nx"], case["ny"]) * case["voxel"] / ph.cyl_radius,
            0.6 * radius / ph.cyl_radius)
    ph.cyl_radius *= k
    ph.spheres = tuple((x * k, y * k, z, r * k) for x, y, z, r in ph.spheres)
    return ph


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _activity(case, seed, frames=1):
    """A positive activity image: the phantom on a warm background, each
    frame with a level of its own."""
    x = _phantom(case, seed).image(_image_params(case), device="cuda") + 0.1
    g = _generator(seed + 1)
    level = 0.5 + torch.rand(frames, 1, 1, 1, generator=g, device="cuda")
    return (x * level).contiguous()


def _sensitivity(case, subsets=1):
    """A sensitivity image as a program loads it from a file: highest on the
    axis, falling towards the rim and the ends, zero outside the FOV."""
    ip = _image_params(case)
    axis = [(torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) / n * 2 - 1
            for n in (ip.nz, ip.ny, ip.nx)]
    z, y, x = torch.meshgrid(*axis, indexing="ij")
    r2 = x * x + y * y
    s = 40.0 * (1.05 - 0.8 * z.abs()) * (1.0 - 0.3 * r2)
    return torch.where(r2 <= 1.0, s, torch.zeros_like(s)).reshape(-1).contiguous()


def _listmode(case, seed):
    """List-mode events on the device, as after reading a file."""
    sc = _scanner(case)
    n = case["events"]
    tof = TOF_FWHM_PS if case.get("tof", True) else None
    ev = synthetic.generate_events(sc, n, seed, phantom=_phantom(case, seed),
                                   tof_fwhm_ps=tof, randoms_fraction=0.1, device="cuda",
                                   chunk=min(1 << 23, max(1 << 17, 2 * n)))
    lm = yrt.ListModeLUT(sc, flagTOF=tof is not None)
    rnd = None
    if case.get("corrections"):
        rnd = 0.02 + 0.02 * torch.rand(n, generator=_generator(seed + 2), device="cuda")
    lm.bind(ev.d1.cpu().numpy().astype(np.uint32), ev.d2.cpu().numpy().astype(np.uint32),
            tof=None if ev.tof is None else ev.tof.cpu().numpy(),
            randoms=None if rnd is None else rnd.cpu().numpy())
    frames = case.get("frames", 1)
    if frames > 1:
        # Frame lengths spread over a factor of ten, events in time order.
        counts = synthetic.frame_counts_loguniform(frames, 1000, 10000, seed + 3)
        edges = np.round(np.cumsum(counts) / counts.sum() * n).astype(np.int64)
        fr = np.searchsorted(edges, np.arange(n), side="right").astype(np.int32)
        lm.setDynamicFrames(np.minimum(fr, frames - 1))
        lm._numDynamicFrames = frames
        if case.get("motion"):
            lm.setMotion(lm.dynamicFrames, synthetic.rigid_transforms(frames, seed + 4))
    lm.device_events()
    return lm


def _projector_params(case, sc):
    pp = yrt.ProjectorParams(sc)
    pp.setProjector(case.get("projector", "S"))
    if case.get("tof"):
        pp.addTOF(TOF_FWHM_PS, TOF_NSTD)
    pp.precision = L.YRTB_COMPENSATED if case["comp"] else L.YRTB_MIRROR
    return pp


def _projection_psf():
    """Gaussian of 4 mm FWHM across the crystals, sampled every 0.5 mm."""
    sig, ks = 4.0 / 2.3548, 0.5
    half = int(np.ceil(3 * sig / ks))
    k = np.exp(-0.5 * ((np.arange(2 * half + 1) - half) * ks / sig) ** 2)
    return 1e9, ks, (k / (k.sum() * ks))[None].astype(np.float32)


def _image_psf(case, variant):
    """The image PSF of a case, and the taps or kernel table it holds."""
    ip = _image_params(case)
    if not variant:
        op = yrt.OperatorPsfDevice.createGaussianFromFWHM(4.5, 4.5, 4.5, ip.vx, ip.vy, ip.vz)
        return op
    # Blurrier away from the centre: 3 x 3 x 2 kernels over the half field.
    op = yrt.OperatorVarPsfDevice(ip)
    half = [0.5 * n * case["voxel"] for n in (ip.nx, ip.ny, ip.nz)]
    kernels = []
    for k in range(2):
        for j in range(3):
            for i in range(3):
                s = case["voxel"] * (0.75 + 0.12 * i + 0.12 * j + 0.1 * k)
                kernels.append(yrt.ConvolutionKernelGaussian(
                    s, s * 1.05, s * 0.95, 4.0, 4.0, 4.0, ip))
    op.setKernelCollection(kernels)
    op.setRangeAndGap(half[0], half[0] / 2, half[1], half[1] / 2, half[2], half[2])
    return op


def prepare(case, seed):
    family = case["family"]
    state = {"case": case}
    if family == "image_psf":
        ip = _image_params(case, case["frames"])
        x = torch.rand(ip.shape, generator=_generator(seed), device="cuda")
        state.update(psf=_image_psf(case, case["variant"]), ip=ip, x=x + 0.1,
                     y=torch.empty_like(x), z=torch.empty_like(x))
        return state
    sc = _scanner(case)
    ip = _image_params(case)
    if family == "project":
        lm = _listmode(case, seed)
        it = lm.getBinIter(case["subsets"], case["subsets"] // 2)
        op = yrt.OperatorProjectorDevice.create(_projector_params(case, sc), it, img_params=ip)
        vals = yrt.ProjectionList(lm)
        vals.allocate()
        w = yrt.ProjectionList(lm)
        w.values = 0.5 + torch.rand(lm.count(), generator=_generator(seed + 5), device="cuda")
        state.update(op=op, x=_activity(case, seed), vals=vals, w=w)
    elif family == "nll":
        lm = _listmode(case, seed)
        state.update(proj=yrt.DeviceProjector(sc, ip, _projector_params(case, sc)),
                     ev=lm.device_events(), x=_activity(case, seed).requires_grad_(True),
                     sens=_sensitivity(case).reshape(ip.shape))
    elif family in ("osem", "lrem"):
        lm = _listmode(case, seed)
        osem = yrt.createOSEM(sc, isLowRank=family == "lrem")
        osem.setImageParams(ip)
        osem.num_MLEM_iterations = case["iterations"]
        osem.num_OSEM_subsets = case["subsets"]
        osem.projectorParams.precision = L.YRTB_COMPENSATED if case["comp"] else L.YRTB_MIRROR
        if case.get("tof", True):
            osem.addTOF(TOF_FWHM_PS, TOF_NSTD)
        osem.setNumRays(case.get("rays", 1))
        osem.setDataInput(lm)
        osem.setSensitivityImages([_sensitivity(case)])
        if case.get("corrections"):
            mu = _phantom(case, seed).mu_image(ip, device="cuda")
            osem.setAttenuationImage(mu, ip)
        if case.get("psf") == "uniform":
            osem.addUniformGaussianImagePSFFromFWHM(4.5, 4.5, 4.5)
        elif case.get("psf") == "variant":
            osem.imagePsf = _image_psf(case, True)
            osem.flagImagePSF = True
        state["osem"] = osem
        if family == "lrem":
            rng = np.random.default_rng(seed + 6)
            t = np.linspace(0, 1, case["frames"])
            H = np.stack([np.exp(-t * r) + 0.2 * rng.random(case["frames"])
                          for r in range(case["rank"])])
            state["H"] = np.ascontiguousarray(H, np.float32)
            g = _generator(seed + 7)
            W = 0.2 + torch.rand((case["rank"],) + ip.shape[1:], generator=g, device="cuda")
            osem.setInitialEstimate(W)
            osem.setUpdateH(case["update_h"])
    elif family in ("histo_osem", "sens"):
        osem = yrt.createOSEM(sc)
        osem.setImageParams(ip)
        osem.projectorParams.precision = L.YRTB_COMPENSATED if case["comp"] else L.YRTB_MIRROR
        if family == "sens":
            osem.setProjector(case["projector"])
            osem.setListModeEnabled(True)
            if case["mu"]:
                osem.setAttenuationImage(_phantom(case, seed).mu_image(ip, device="cuda"), ip)
            h = yrt.Histogram3D(sc)
            g = _generator(seed)
            h.data = (0.8 + 0.4 * torch.rand(h.histoSize, generator=g, device="cuda")).cpu().numpy()
            osem.setSensitivityHistogram(h)
        else:
            osem.setProjector("DD")
            osem.projectorParams.setProjPsf(*_projection_psf())
            osem.num_MLEM_iterations = case["iterations"]
            osem.num_OSEM_subsets = case["subsets"]
            osem.setDataInput(yrt.convertToHistogram3D(_listmode(dict(case, tof=False), seed)))
            osem.setSensitivityImages([_sensitivity(case)] * case["subsets"])
        state["osem"] = osem
    elif family == "histo_op":
        h = yrt.Histogram3D(sc)
        it = h.getBinIter(case["subsets"], case["subsets"] - 1)
        op = yrt.OperatorProjectorDevice.create(_projector_params(case, sc), it, img_params=ip)
        vals = yrt.ProjectionList(h)
        vals.allocate()
        w = yrt.ProjectionList(h)
        w.values = 0.5 + torch.rand(h.count(), generator=_generator(seed), device="cuda")
        state.update(op=op, x=_activity(case, seed), vals=vals, w=w)
    else:
        raise ValueError(family)
    return state


# --------------------------------------------------------------------- pass --
def run(state):
    family = state["case"]["family"]
    if family == "image_psf":
        state["psf"].applyA(state["x"], state["y"], state["ip"])
        state["psf"].applyAH(state["x"], state["z"], state["ip"])
        return {"A": state["y"], "AH": state["z"]}
    if family in ("project", "histo_op"):
        img = torch.zeros_like(state["x"])
        state["op"].applyA(state["x"], state["vals"])
        state["op"].applyAH(state["w"], img)
        return {"A": state["vals"].values, "AH": img}
    if family == "nll":
        x = state["x"]
        x.grad = None
        loss = poisson_nll_fused(x, state["proj"], state["ev"], state["sens"])
        loss.backward()
        return {"loss": loss.detach(), "grad": x.grad}
    osem = state["osem"]
    if family == "sens":
        return {"sens": osem.generateSensitivityImages()}
    if family == "lrem":
        H = state["H"].copy()
        osem.setHBasisFromNumpy(H)
        W = osem.reconstruct()
        return {"W": W, "H": H}
    return {"image": osem.reconstruct()}


# --------------------------------------------------------------------- work --
def _crossings(case):
    """Mean voxels a line crosses: about 1.3 per voxel length of the part of
    the line inside the grid (and the TOF window)."""
    length = 0.9 * min(case["nx"], case["ny"]) * case["voxel"]
    if case.get("tof") or case["family"] == "lrem":
        sigma = TOF_FWHM_PS * 0.299792458 * 0.5 / 2.3548
        length = min(length, 2 * TOF_NSTD * sigma)
    return 1.3 * length / case["voxel"]


def _bins(case):
    axial, _, _, _, _, dpr, rings, _, mrd, mad, _ = SCANNERS[case["scanner"]]
    nz = (mrd + 1) * rings - mrd * (mrd + 1) // 2
    return (2 * nz - rings) * dpr * (dpr // 2 + 1 - mad)


def work(case):
    """Inputs read once and results written once per pass over the data, and
    about 12 operations per voxel a line crosses and direction."""
    J = case["nx"] * case["ny"] * case["nz"]
    family = case["family"]
    if family == "image_psf":
        n = J * case["frames"]
        taps = 125 if case["variant"] else 15
        return {"bytes": 12.0 * n, "flops": 4.0 * n * taps}
    if family == "histo_op":
        n = _bins(case) // case["subsets"]
        return {"bytes": 8.0 * n + 8.0 * J, "flops": 24.0 * n * _crossings(case)}
    if family == "sens":
        n = _bins(case)
        per = 24.0 if case["mu"] else 12.0
        return {"bytes": 4.0 * n + 8.0 * J, "flops": per * n * _crossings(case)}
    if family == "histo_osem":
        n = min(_bins(case), case["events"]) * 0.25
        per = 2 * 18.0 * 0.8 * min(case["nx"], case["ny"])
        return {"bytes": 4.0 * _bins(case) + 16.0 * J * case["subsets"],
                "flops": 4.0 * n * per * case["iterations"]}
    n = case["events"]
    row = 12.0 if case.get("tof") or family == "lrem" else 8.0
    if family == "project":
        n = n / case["subsets"]
        return {"bytes": (row + 4.0) * 2 * n + 8.0 * J, "flops": 24.0 * n * _crossings(case)}
    if family == "nll":
        return {"bytes": row * n + 12.0 * J, "flops": 24.0 * n * _crossings(case)}
    T = case.get("frames", 1)
    passes = case["iterations"]
    flops = 24.0 * n * _crossings(case) * passes * case.get("rays", 1)
    nbytes = row * n * passes + 16.0 * J * T * passes * case["subsets"]
    if family == "lrem":
        nbytes += 4.0 * J * case["rank"] * 2 * passes * case["subsets"]
        flops += 4.0 * J * case["rank"] * T * passes * case["subsets"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Relative error (2-norm) between two correct FP32 implementations:
    one pass over the data sums in 32 bits in any order; a reconstruction
    carries such differences through its updates."""
    family = case["family"]
    if family in ("osem", "histo_osem", "lrem"):
        return {"rel": 2e-4, "max": 0.03}
    return {"rel": 2e-5, "max": 2e-3}


# ------------------------------------------------------------ 64-bit values --
def _lut(case):
    """Crystal centres and orientations: the scanner's look-up table, an input."""
    lut = torch.from_numpy(_scanner(case).createLUT()).cuda().double()
    return lut[:, :3].contiguous(), lut[:, 3:].contiguous()


def _slab(p, d, lo, hi, amin, amax):
    """Narrows [amin, amax] to the part of p + a d between lo and hi."""
    flat = d == 0
    inv = 1.0 / torch.where(flat, torch.ones_like(d), d)
    a, b = (lo - p) * inv, (hi - p) * inv
    miss = flat & ((p < lo) | (p > hi))
    near = torch.where(flat, torch.zeros_like(p), torch.minimum(a, b))
    far = torch.where(flat, torch.where(miss, -torch.ones_like(p), torch.ones_like(p)),
                      torch.maximum(a, b))
    return torch.maximum(amin, near), torch.minimum(amax, far)


def _tof_constants():
    sigma = float(np.float32(TOF_FWHM_PS * 0.299792458 * 0.5 / (2 * math.sqrt(2 * math.log(2)))))
    return sigma, TOF_NSTD * sigma, 1.0 / (math.sqrt(2 * math.pi) * sigma)


def _siddon64(case, p1, p2, tof):
    """Voxel offsets (N, M) and weights (N, M) of the lines p1 -> p2: the
    lengths between consecutive plane crossings inside the grid, the
    cylinder that fits it and the TOF window, times the TOF Gaussian at each
    piece's centre."""
    n = [case["nx"], case["ny"], case["nz"]]
    v = case["voxel"]
    ln = [k * v for k in n]
    d = p2 - p1
    norm = d.norm(dim=1)
    radius = max(ln[0], ln[1]) / 2 - v / 1000.0
    A = d[:, 0] ** 2 + d[:, 1] ** 2
    B = 2 * (d[:, 0] * p1[:, 0] + d[:, 1] * p1[:, 1])
    C = p1[:, 0] ** 2 + p1[:, 1] ** 2 - radius * radius
    disc = B * B - 4 * A * C
    sq = disc.clamp_min(0).sqrt()
    one = torch.ones_like(A)
    amin = torch.where(A > 0, (-B - sq) / (2 * A), 0 * one).clamp_min(0)
    amax = torch.where(A > 0, (-B + sq) / (2 * A), one).clamp_max(1)
    amax = torch.where(disc <= 0, -one, amax)
    for k in range(3):
        amin, amax = _slab(p1[:, k], d[:, k], -ln[k] / 2, ln[k] / 2, amin, amax)
    if tof is not None:
        sigma, trunc, gain = _tof_constants()
        centre = tof.double() * float(np.float32(0.299792458)) * 0.5
        amin = torch.maximum(amin, 0.5 + (centre - trunc) / norm)
        amax = torch.minimum(amax, 0.5 + (centre + trunc) / norm)
    live = amin < amax
    amax = torch.where(live, amax, amin)
    cuts = [amin[:, None], amax[:, None]]
    for k in range(3):
        planes = torch.arange(n[k] + 1, device=p1.device, dtype=torch.float64) * v - ln[k] / 2
        inv = torch.where(d[:, k] == 0, torch.full_like(norm, math.inf), 1.0 / d[:, k])
        a = (planes[None] - p1[:, k:k + 1]) * inv[:, None]
        a = torch.where(torch.isfinite(a), a, amin[:, None])
        cuts.append(torch.minimum(torch.maximum(a, amin[:, None]), amax[:, None]))
    a = torch.cat(cuts, 1).sort(dim=1).values
    seg = a[:, 1:] - a[:, :-1]
    mid = 0.5 * (a[:, 1:] + a[:, :-1])
    off = torch.zeros_like(mid, dtype=torch.int64)
    for k, step in ((2, n[0] * n[1]), (1, n[0]), (0, 1)):
        i = torch.floor((p1[:, k:k + 1] + mid * d[:, k:k + 1] + ln[k] / 2) / v).long()
        off += i.clamp(0, n[k] - 1) * step
    w = seg * norm[:, None] * live[:, None]
    if tof is not None:
        pc = 0.5 * norm + centre
        w = w * torch.exp(-0.5 * ((mid * norm[:, None] - pc[:, None]) / sigma) ** 2) * gain
    return off, w


def _kernel_integral(x, taps, step):
    """Integral up to x of the kernel with these taps (linear between them,
    zero beyond one step from the ends)."""
    half = (taps.numel() - 1) // 2
    v = torch.nn.functional.pad(taps, (2, 3))
    bins = 0.5 * step * (v[:-1] + v[1:])
    total = torch.cat([torch.zeros_like(bins[:1]), bins.cumsum(0)])
    s = (x / step + half + 2).clamp(0, v.numel() - 1.001)
    i = s.floor().long()
    t = s - i
    return total[i] + step * (v[i] * t + 0.5 * (v[i + 1] - v[i]) * t * t)


def _dd64(case, p1, p2, n1, n2, tof, psf):
    """Distance-driven footprint: voxel offsets and weights (N, rows * K * Kz)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    v = case["voxel"]
    lx, ly, lz = nx * v, ny * v, nz * v
    _, thick_z, thick_t = SCANNERS[case["scanner"]][:3]
    d = p2 - p1
    norm = d.norm(dim=1)
    amin, amax = torch.zeros_like(norm), torch.ones_like(norm)
    for k, ext in ((0, lx), (1, ly), (2, lz)):
        amin, amax = _slab(p1[:, k], d[:, k], -0.5 * (ext - v), 0.5 * (ext - v), amin, amax)
    if tof is not None:
        sigma, trunc, gain = _tof_constants()
        centre = tof.double() * float(np.float32(0.299792458)) * 0.5
        amin = torch.maximum(amin, 0.5 + (centre - trunc) / norm)
        amax = torch.minimum(amax, 0.5 + (centre + trunc) / norm)
    y_main = d[:, 1].abs() > d[:, 0].abs()
    pick = lambda t: torch.where(y_main, t[:, 1], t[:, 0])
    other = lambda t: torch.where(y_main, t[:, 0], t[:, 1])
    n_main = torch.where(y_main, ny, nx)
    n_other = torch.where(y_main, nx, ny)
    row0 = torch.floor((pick(p1) + amin * pick(d)) / v + 0.5 * n_main)
    row1 = torch.floor((pick(p1) + amax * pick(d)) / v + 0.5 * n_main)
    lo = torch.minimum(row0, row1).clamp_min(0)
    hi = torch.minimum(torch.maximum(row0, row1), n_main - 1.0)
    rows = torch.arange(max(nx, ny), device=p1.device, dtype=torch.float64)[None]
    row_ok = (rows >= lo[:, None]) & (rows <= hi[:, None])
    pix = -0.5 * v * n_main[:, None] + (rows + 0.5) * v

    def edges(c, o):
        xy2 = o[:, 0] ** 2 + o[:, 1] ** 2
        xy = xy2.sqrt()
        t = torch.stack([o[:, 1] / xy, -o[:, 0] / xy], 1)
        zn = ((o[:, 0] * o[:, 2]) ** 2 + (o[:, 1] * o[:, 2]) ** 2 + xy2).sqrt()
        return t, pick(o) * o[:, 2] / zn, -xy2 / zn

    t1, zi1, zz1 = edges(p1, n1)
    t2, zi2, zz2 = edges(p2, n2)
    h = 0.5 * thick_t
    hz = 0.5 * thick_z

    def line(a_main, a_val, b_main, b_val):
        s = (pix - a_main[:, None]) / (b_main - a_main)[:, None]
        return a_val[:, None] + s * (b_val - a_val)[:, None]

    side = lambda p, t, s: p[:, :2] + s * h * t
    e1, e2 = {s: side(p1, t1, s) for s in (-1, 1)}, {s: side(p2, t2, s) for s in (-1, 1)}
    r0 = line(pick(e1[-1]), other(e1[-1]), pick(e2[1]), other(e2[1]))
    r1 = line(pick(e1[1]), other(e1[1]), pick(e2[-1]), other(e2[-1]))
    r0, r1 = torch.minimum(r0, r1), torch.maximum(r0, r1)
    z0 = line(pick(p1) - hz * zi1, p1[:, 2] - hz * zz1, pick(p2) - hz * zi2, p2[:, 2] - hz * zz2)
    z1 = line(pick(p1) + hz * zi1, p1[:, 2] + hz * zz1, pick(p2) + hz * zi2, p2[:, 2] + hz * zz2)
    z0, z1 = torch.minimum(z0, z1), torch.maximum(z0, z1)
    ext = 0.0
    if psf is not None:
        step, taps = psf
        ext = ((taps.numel() + 1) // 2) * step
    off_o = 0.5 * (n_other - 1)[:, None]
    i0 = torch.round((r0 - ext) / v + off_o).clamp_min(0)
    i1 = torch.minimum(torch.round((r1 + ext) / v + off_o), n_other[:, None] - 1.0)
    k0 = torch.round(z0 / v + 0.5 * (nz - 1)).clamp_min(0)
    k1 = torch.round(z1 / v + 0.5 * (nz - 1)).clamp_max(nz - 1)
    K = max(1, int(torch.where(row_ok, i1 - i0, 0).max()) + 1)
    Kz = max(1, int(torch.where(row_ok, k1 - k0, 0).max()) + 1)
    j = i0[..., None] + torch.arange(K, device=p1.device)
    a = -0.5 * v * n_other[:, None, None] + j * v
    b = a + v
    R0, R1 = r0[..., None], r1[..., None]
    ok = (j <= i1[..., None]) & (R1 + ext >= a) & (R0 - ext < b) & row_ok[..., None]
    if psf is None:
        wt = torch.minimum(b, R1) - torch.maximum(a, R0)
    else:
        xa, xb = a - R1, b - R0
        wt = _kernel_integral(xb, taps, step) - _kernel_integral(xa, taps, step)
        wt = torch.where((xa > ext) | (xb < -ext), 0.0, wt)
    cosine = (pick(d).abs() / norm)[:, None, None]
    wt = torch.where(ok, wt / (R1 - R0) * v / cosine, 0.0)
    if tof is not None:
        s = (pix - pick(p1)[:, None]) / pick(d)[:, None]
        x = (s * norm[:, None] - (0.5 * norm + centre)[:, None]) / sigma
        wt = wt * (torch.exp(-0.5 * x * x) * gain)[..., None]
    q = k0[..., None] + torch.arange(Kz, device=p1.device)
    qa = -0.5 * lz + q * v
    Z0, Z1 = z0[..., None], z1[..., None]
    okz = (q <= k1[..., None]) & (Z1 >= qa) & (Z0 < qa + v)
    wz = torch.where(okz, (torch.minimum(qa + v, Z1) - torch.maximum(qa, Z0)) / (Z1 - Z0), 0.0)
    w = wt[..., None] * wz[:, :, None, :]
    ym = y_main[:, None, None]
    rr = rows[..., None].expand_as(j)
    flat = torch.where(ym, nx * rr + j, nx * j + rr)
    off = (q[:, :, None, :] * (nx * ny) + flat[..., None]).long().clamp(0, nx * ny * nz - 1)
    N = p1.shape[0]
    return off.reshape(N, -1), torch.where(w != 0, w, 0.0).reshape(N, -1)


class _Lines:
    """The lines of a case in 64 bits, walked in chunks."""

    def __init__(self, case, d1, d2, tof=None, frame=None, motion=None, psf=None):
        pos, ori = _lut(case)
        self.case, self.d1, self.d2 = case, d1.long(), d2.long()
        self.pos, self.ori = pos, ori
        self.tof, self.frame, self.motion, self.psf = tof, frame, motion, psf
        self.dd = case.get("projector", "S") == "DD" or case["family"] == "histo_osem"
        rows = max(case["nx"], case["ny"])
        self.width = rows * 40 if self.dd else case["nx"] + case["ny"] + case["nz"] + 5
        self.chunk = max(1000, int(4e7 / self.width))

    def cost(self, passes=1):
        return float(self.d1.numel()) * self.width * passes

    def walk(self, sel):
        p1, p2 = self.pos[self.d1[sel]], self.pos[self.d2[sel]]
        if self.motion is not None:
            m = self.motion.double()[self.frame[sel].long()].reshape(-1, 3, 4)
            move = lambda p: (m[:, :, :3] @ p[:, :, None])[:, :, 0] + m[:, :, 3]
            p1, p2 = move(p1), move(p2)
        t = None if self.tof is None else self.tof[sel]
        if self.dd:
            return _dd64(self.case, p1, p2, self.ori[self.d1[sel]], self.ori[self.d2[sel]],
                         t, self.psf)
        return _siddon64(self.case, p1, p2, t)

    def chunks(self, index):
        for k in range(0, index.numel(), self.chunk):
            sel = index[k:k + self.chunk]
            off, w = self.walk(sel)
            if self.frame is not None:
                J = self.case["nx"] * self.case["ny"] * self.case["nz"]
                off = off + self.frame[sel].long()[:, None] * J
            yield k, sel, off, w


def _blur64(case, x, kernels, adjoint):
    """Separable circular convolution of (frames, nz, ny, nx)."""
    for dim, k in ((3, kernels[0]), (2, kernels[1]), (1, kernels[2])):
        c = len(k) // 2
        y = torch.zeros_like(x)
        for t in range(-c, c + 1):
            y += float(k[t + c]) * torch.roll(x, -t if adjoint else t, dim)
        x = y
    return x


def _var_blur64(case, x, op, adjoint):
    """Every voxel's own kernel, the table's nearest to its distance from the
    centre along each axis: gathered, or (adjoint) scattered."""
    v = case["voxel"]
    gaps = [float(t) for t in op._gap]
    lut = [int(float(r) / g) + 1 for r, g in zip(op._range, gaps)]
    axis = []
    for n, g, m in zip((case["nx"], case["ny"], case["nz"]), gaps, lut):
        c = ((torch.arange(n, device="cuda") + 0.5) * v - n * v / 2).abs()
        # Half-way distances go to the farther kernel, as round() does.
        axis.append(torch.floor(c.float() / g + 0.5).long().clamp_max(m - 1))
    which = (axis[0][None, None] + lut[0] * (axis[1][None, :, None] +
                                             lut[1] * axis[2][:, None, None]))
    out = torch.zeros_like(x)
    for k, kernel in enumerate(op._kernels):
        mine = (which == k)[None]
        if not bool(mine.any()):
            continue
        w = kernel.weights
        cz, cy, cx = (s // 2 for s in w.shape)
        src = torch.where(mine, x, 0.0) if adjoint else x
        part = torch.zeros_like(x)
        for dz in range(-cz, cz + 1):
            for dy in range(-cy, cy + 1):
                for dx in range(-cx, cx + 1):
                    s = (dz, dy, dx) if adjoint else (-dz, -dy, -dx)
                    part += float(w[dz + cz, dy + cy, dx + cx]) * torch.roll(src, s, (1, 2, 3))
        out += part if adjoint else torch.where(mine, part, 0.0)
    return out


def _em_pass64(lines, index, x, total, factor, additive, em, meas=None):
    """em += A^T (factor m / (factor A x + additive)) over the items index."""
    for k, sel, off, w in lines.chunks(index):
        u = (w * x[off]).sum(1)
        a = 1.0 if factor is None else factor[sel]
        u = u * a
        if additive is not None:
            u = u + additive[sel].double()
        m = 1.0 if meas is None else meas[k:k + sel.numel()].double()
        ratio = torch.where(u.abs() > DENOM_THRESHOLD, m / u, 0.0) * a
        em.index_add_(0, off.reshape(-1), (w * ratio[:, None]).reshape(-1))


def _attenuation64(case, lines, mu, index):
    plain = _Lines(dict(case, projector="S", family="osem"), lines.d1, lines.d2,
                   frame=lines.frame, motion=lines.motion)
    flat = mu.double().reshape(-1)
    out = torch.empty(lines.d1.numel(), dtype=torch.float64, device="cuda")
    for k in range(0, index.numel(), plain.chunk):
        sel = index[k:k + plain.chunk]
        off, w = plain.walk(sel)
        out[sel] = torch.exp(-0.1 * (w * flat[off]).sum(1))
    return out


def _histogram_pairs(case, bins):
    """Crystal pairs of histogram bins (z bin, phi, r), and which are valid."""
    _, _, _, _, _, dpr, rings, _, mrd, mad, _ = SCANNERS[case["scanner"]]
    num_r = dpr // 2 + 1 - mad
    cut = mad // 2 + (1 if mad % 2 and dpr % 4 == 0 else 0)
    zb, phi, r = bins // (dpr * num_r), bins % (dpr * num_r) // num_r, bins % num_r
    half = torch.where(phi % 2 != 0, dpr // 2 + 1, dpr // 2)
    a = r - dpr // 4 + cut
    b = half - a
    a = (torch.where(a < 0, a + dpr, a) + phi // 2) % dpr
    b = (torch.where(b < 0, b + dpr, b) + phi // 2) % dpr
    a, b = torch.minimum(a, b), torch.maximum(a, b)
    z1, z2 = [list(range(rings))], [list(range(rings))]
    for dz in range(1, mrd + 1):
        z1.append(list(range(rings - dz)))
        z2.append(list(range(dz, rings)))
    up1, up2 = sum(z1[1:], []), sum(z2[1:], [])
    tz1 = torch.tensor(z1[0] + up1 + up2, device=bins.device)
    tz2 = torch.tensor(z2[0] + up2 + up1, device=bins.device)
    return a + tz1[zb] * dpr, b + tz2[zb] * dpr, a != b


def _subset_bins(case, subsets, subset):
    dpr, mad = SCANNERS[case["scanner"]][5], SCANNERS[case["scanner"]][9]
    num_r = dpr // 2 + 1 - mad
    bins = torch.arange(_bins(case), device="cuda")
    return bins[(bins // num_r) % dpr % subsets == subset]


#: Weights that exact() may compute in about 20 seconds.
EXACT_MOST = 6e9


def exact(case, seed):
    family = case["family"]
    J = case["nx"] * case["ny"] * case["nz"]
    shape = (1, case["nz"], case["ny"], case["nx"])
    if family == "image_psf":
        s = prepare(case, seed)
        x = s["x"].double()
        if case["variant"]:
            return {"A": _var_blur64(case, x, s["psf"], False),
                    "AH": _var_blur64(case, x, s["psf"], True)}
        k = (s["psf"].getKernelX(), s["psf"].getKernelY(), s["psf"].getKernelZ())
        return {"A": _blur64(case, x, k, False), "AH": _blur64(case, x, k, True)}
    if case.get("rays", 1) > 1:
        return None  # the extra rays' offsets are a random stream of the projector's own
    if family == "histo_op":
        bins = _subset_bins(case, case["subsets"], case["subsets"] - 1)
        d1, d2, ok = _histogram_pairs(case, bins)
        lines = _Lines(case, d1, d2)
        if lines.cost(2) > EXACT_MOST:
            return None
        s = prepare(case, seed)
        x = s["x"].double().reshape(-1)
        vals = torch.zeros(_bins(case), dtype=torch.float64, device="cuda")
        img = torch.zeros(J, dtype=torch.float64, device="cuda")
        w_in = s["w"].values.double()[bins]
        for _, sel, off, w in lines.chunks(torch.arange(bins.numel(), device="cuda")):
            vals[bins[sel]] = (w * x[off]).sum(1)
            img.index_add_(0, off.reshape(-1), (w * w_in[sel][:, None]).reshape(-1))
        return {"A": vals, "AH": img.reshape(shape)}
    if family == "sens":
        bins = _subset_bins(case, 1, 0)
        d1, d2, ok = _histogram_pairs(case, bins)
        lines = _Lines(case, d1[ok], d2[ok])
        if lines.cost(2 if case["mu"] else 1) > EXACT_MOST:
            return None
        osem = prepare(case, seed)["osem"]
        v = torch.from_numpy(osem._sens_histo.data).cuda().double()[bins[ok]]
        index = torch.arange(v.numel(), device="cuda")
        if case["mu"]:
            v = v * _attenuation64(case, lines, osem._att_image, index)
        img = torch.zeros(J, dtype=torch.float64, device="cuda")
        for _, sel, off, w in lines.chunks(index):
            img.index_add_(0, off.reshape(-1), (w * v[sel][:, None]).reshape(-1))
        return {"sens": [torch.where(img <= osem.hardThreshold, 0.0, img)]}
    if family == "histo_osem":
        s = prepare(case, seed)
        osem = s["osem"]
        data = torch.from_numpy(osem.getDataInput().data).cuda()
        bins = torch.nonzero(data).reshape(-1)
        d1, d2, ok = _histogram_pairs(case, bins)
        bins, d1, d2 = bins[ok], d1[ok], d2[ok]
        step, taps = _projection_psf()[1:]
        psf = (step, torch.from_numpy(taps[0]).cuda().double())
        lines = _Lines(case, d1, d2, psf=psf)
        if lines.cost(case["iterations"]) > EXACT_MOST:
            return None
        dpr, mad = SCANNERS[case["scanner"]][5], SCANNERS[case["scanner"]][9]
        sub = (bins // (dpr // 2 + 1 - mad)) % dpr % case["subsets"]
        sens = _sensitivity(case).double()
        x = torch.where(sens > 0, 0.125, 0.0).double()
        for _ in range(case["iterations"]):
            for k in range(case["subsets"]):
                index = torch.nonzero(sub == k).reshape(-1)
                em = torch.zeros_like(x)
                _em_pass64(lines, index, x, J, None, None, em, meas=data[bins[index]])
                x = torch.where(sens > EPS_FLT, x * (em / sens), x)
        return {"image": x.reshape(shape)}
    # List-mode families.
    passes = {"project": 2, "nll": 1}.get(family, case.get("iterations", 1))
    n = case["events"]
    probe = _Lines(case, torch.empty(0), torch.empty(0))
    if n * probe.width * (passes + (1 if case.get("corrections") else 0)) > EXACT_MOST:
        return None
    s = prepare(case, seed)
    lm = (s["osem"].getDataInput() if "osem" in s else
          s["vals"].reference if "vals" in s else _listmode(case, seed))
    ev = lm.device_events()
    lines = _Lines(case, ev.d1, ev.d2, tof=ev.tof, frame=ev.frame, motion=ev.motion)
    every = torch.arange(n, device="cuda")
    if family == "project":
        it = s["op"].getBinIter()
        index = every[it.idxSubset::it.numSubsets]
        x = s["x"].double().reshape(-1)
        vals = torch.zeros(n, dtype=torch.float64, device="cuda")
        img = torch.zeros(J, dtype=torch.float64, device="cuda")
        w_in = s["w"].values.double()
        for _, sel, off, w in lines.chunks(index):
            vals[sel] = (w * x[off]).sum(1)
            img.index_add_(0, off.reshape(-1), (w * w_in[sel][:, None]).reshape(-1))
        return {"A": vals, "AH": img.reshape(shape)}
    if family == "nll":
        x = s["x"].detach().double().reshape(-1)
        sens = s["sens"].double().reshape(-1)
        loss = (sens * x).sum()
        bp = torch.zeros_like(x)
        for _, sel, off, w in lines.chunks(every):
            u = (w * x[off]).sum(1)
            loss = loss - torch.log(u.clamp_min(1e-12)).sum()
            r = torch.where(u > 1e-12, 1.0 / u, 0.0)
            bp.index_add_(0, off.reshape(-1), (w * r[:, None]).reshape(-1))
        return {"loss": loss, "grad": (sens - bp).reshape(shape)}
    osem = s["osem"]
    T, S = case["frames"], case["subsets"]
    full = _sensitivity(case).double()
    sens = full / S
    factor = None
    if case.get("corrections"):
        factor = _attenuation64(case, lines, osem._att_image, every)
    vol = (T,) + shape[1:]
    if family == "osem":
        x = torch.where(full > 0, 0.125, 0.0).double().repeat(T)
        for _ in range(case["iterations"]):
            for k in range(S):
                em = torch.zeros_like(x)
                src = x
                if case["psf"] == "uniform":
                    op = osem.imagePsf
                    ker = (op.getKernelX(), op.getKernelY(), op.getKernelZ())
                    src = _blur64(case, x.reshape(vol), ker, False).reshape(-1)
                elif case["psf"] == "variant":
                    src = _var_blur64(case, x.reshape(vol), osem.imagePsf, False).reshape(-1)
                _em_pass64(lines, every[k::S], src, J, factor, ev.additive, em)
                if case["psf"] == "uniform":
                    em = _blur64(case, em.reshape(vol), ker, True).reshape(-1)
                elif case["psf"] == "variant":
                    em = _var_blur64(case, em.reshape(vol), osem.imagePsf, True).reshape(-1)
                x = torch.where(sens > EPS_FLT, x.reshape(T, J) * (em.reshape(T, J) / sens),
                                x.reshape(T, J)).reshape(-1)
        return {"image": x.reshape(vol)}
    # lrem: rank images W, basis H.
    H = torch.from_numpy(s["H"]).cuda().double()
    R = case["rank"]
    W = osem._initial.double().reshape(R, J) * (full > 0)
    c = (W * sens).sum(1) if case["update_h"] else H.sum(1)
    for _ in range(case["iterations"]):
        for k in range(S):
            X = (H.t() @ W).reshape(-1)
            E = torch.zeros_like(X)
            _em_pass64(lines, every[k::S], X, J, None, None, E)
            E = E.reshape(T, J)
            if case["update_h"]:
                H = H * ((W @ E.t()) / c.clamp_min(EPS_FLT)[:, None])
            else:
                Wn = (H @ E) / c[:, None]
                W = torch.where(sens > EPS_FLT / c[:, None], W * (Wn / sens), W)
    return {"W": W.reshape((R,) + shape[1:]), "H": H}
