"""Workloads for timing the projectors and the reconstruction loops through the package's
public entry points.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more
of the same ranges, ``prepare(case, seed)`` the inputs and the system matrix a program holds
before the call, ``run(state)`` one pass, ``work(case)`` the bytes and operations a pass
cannot do without and ``exact(case, seed)`` the values of a pass in 64 bits, restated in
plain torch.

All data are synthetic and made from the seed alone: ellipsoid phantoms with hot spheres,
Poisson counts of their analytic line integrals (SPECT) and listmode events emitted by them
(PET).  Units are those of the package: cm for SPECT, mm for PET.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

DELTA = 1e-11  # the package's guard in divisions and logarithms


# ------------------------------------------------------------------------------- cases
def _spect(name, op, n, nz, angles, subsets, *, psf, voxel=0.442, radius=22.0, orbit=0.0,
           scatter=False, batch=1):
    c = {"path": "spect", "op": op, "n": n, "nz": nz, "angles": angles, "subsets": subsets,
         "psf": psf, "voxel": voxel, "radius": radius, "orbit": orbit, "scatter": scatter,
         "batch": batch}
    return {"name": name, **c} if name else c


def _serving(name, mix, subsets):
    """``mix``: 'size x angles' of every reconstruction, comma separated."""
    c = {"path": "serving", "mix": mix, "subsets": subsets, "voxel": 0.442, "radius": 22.0}
    return {"name": name, **c} if name else c


def _pet(name, path, op, nx, nz, voxel, crystals, rings, subsets, *, events=0, bins=0):
    c = {"path": path, "op": op, "nx": nx, "nz": nz, "voxel": voxel, "crystals": crystals,
         "rings": rings, "subsets": subsets, "events": events, "bins": bins}
    return {"name": name, **c} if name else c


def listed():
    return [
        # One attenuated projection of a small SPECT study, one subset: the smallest call of a
        # program that writes its own loop over system_matrix.forward.
        _spect("spect_att_64_forward", "forward", 64, 64, 64, 8, psf=False, voxel=0.48,
               radius=25.0),
        # A whole OSEM iteration (8 sub-iterations) of that study: launches and host time count.
        _spect("spect_att_64_osem", "osem", 64, 64, 64, 8, psf=False, voxel=0.48, radius=25.0),
        # The projector of the usual clinical study (attenuation and collimator response), one
        # subset, in both directions: what every algorithm outside the package is built on.
        _spect("spect_psf_128_forward", "forward", 128, 128, 120, 10, psf=True),
        _spect("spect_psf_128_backward", "backward", 128, 128, 120, 10, psf=True),
        # One OSEM iteration (10 sub-iterations) of that study: the benchmark's own workload.
        _spect("spect_psf_128_osem", "osem", 128, 128, 120, 10, psf=True),
        # A cropped field of view with odd extents, a body-contour orbit and a scatter estimate:
        # one OSEM iteration where no extent is a multiple of anything.
        _spect("spect_psf_ragged_osem", "osem", 101, 83, 45, 5, psf=True, orbit=4.0,
               scatter=True),
        # Penalised reconstruction of the clinical study: one BSREM iteration with the
        # relative-difference prior.
        _spect("spect_psf_128_bsrem", "bsrem", 128, 128, 120, 10, psf=True, scatter=True),
        # Gradient of the Poisson likelihood with respect to a small batch of objects over all
        # angles, as a learned reconstruction takes it (autograd, exact adjoint).
        _spect("spect_psf_128_gradient", "gradient", 128, 128, 120, 1, psf=True, batch=2),
        # A server's batch: independent studies of uneven sizes, one OSEM iteration of all.
        _serving("spect_serving_uneven", "64x60,128x120,96x90,64x120,128x60,96x60", 10),
        # TOF listmode projection of one subset's events on a 600-crystal, 96-ring scanner.
        _pet("pet_lm_tof_forward", "pet_lm", "forward", 200, 96, 2.0, 600, 96, 4,
             events=2_000_000, bins=13),
        # One TOF listmode OSEM iteration over the same events (4 sub-iterations).
        _pet("pet_lm_tof_osem", "pet_lm", "osem", 200, 96, 2.0, 600, 96, 4, events=2_000_000,
             bins=13),
        # Sinogram back projection of one subset of angles, no TOF, on a smaller scanner.
        _pet("pet_sino_backward", "pet_sino", "backward", 128, 48, 4.0, 300, 24, 10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["att", "psf", "psf", "psf", "psf", "serving", "pet_lm", "pet_lm", "pet_sino"])
    if kind in ("att", "psf"):
        psf = kind == "psf"
        n = rng.choice([64, 96, 128, rng.randint(32, 140), rng.randint(32, 140)])
        nz = rng.choice([n, 64, 128, rng.randint(16, 140)])
        subsets = rng.randint(4, 12)
        angles = rng.choice([60, 90, 120, rng.randint(30, 128)])
        op = rng.choice(["forward", "backward", "osem", "bsrem", "gradient"])
        batch = rng.randint(1, 2) if op == "gradient" else 1
        if op in ("osem", "bsrem", "gradient"):
            angles = min(angles, 90)
        voxel = round(rng.uniform(0.4, 0.5), 3)
        return _spect(None, op, n, nz, angles, 1 if op == "gradient" else min(subsets, angles),
                      psf=psf, voxel=voxel, radius=round(rng.uniform(20.0, 26.0), 1),
                      orbit=rng.choice([0.0, round(rng.uniform(1.0, 4.0), 1)]),
                      scatter=op in ("osem", "bsrem") and rng.random() < 0.5, batch=batch)
    if kind == "serving":
        mix = ",".join(f"{rng.choice([64, 96, 128])}x{rng.choice([60, 90, 120])}"
                       for _ in range(rng.randint(2, 6)))
        return _serving(None, mix, rng.randint(6, 10))
    bins = rng.choice([0, 13, rng.randint(7, 25)])
    nx = rng.randint(64, 200)
    if kind == "pet_lm":
        return _pet(None, kind, rng.choice(["forward", "backward", "osem"]), nx,
                    rng.randint(24, 96), round(400.0 / nx, 2), rng.choice([300, 480, 600]),
                    rng.randint(16, 96), rng.randint(2, 8), events=_log(rng, 20_000, 2_000_000),
                    bins=bins)
    return _pet(None, kind, rng.choice(["forward", "backward"]), min(nx, 128),
                rng.randint(24, 48), round(512.0 / min(nx, 128), 2),
                rng.choice([180, 240, 300]), rng.randint(8, 20),
                rng.randint(15, 30) if bins else rng.randint(10, 30), bins=bins)


# ------------------------------------------------------------------------- SPECT inputs
def _gen(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed))


def _uniform(shape, lo, hi, gen, device):
    r = torch.rand(shape, generator=gen, device=device, dtype=torch.float64)
    return lo + (hi - lo) * r


def _angles(c):
    return torch.linspace(0, 360, c["angles"] + 1, dtype=torch.float64)[:-1].to(torch.float32)


def _radii(c):
    """Detector radius of every angle (cm): a circle, or an ellipse-like orbit in a few steps."""
    if not c["orbit"]:
        return [float(c["radius"])] * c["angles"]
    t = _angles(c).double() * math.pi / 180
    r = c["radius"] + c["orbit"] * torch.cos(2 * t)
    return [float(v) for v in torch.round(r * 2) / 2]


def _ellipsoids(c, gen, device):
    """Rows (activity, x, y, z, rx, ry, rz) of a body and three hot spheres, in cm."""
    e = c["n"] * c["voxel"] / 2
    ez = c["nz"] * c["voxel"] / 2
    u = _uniform((3, 4), 0.0, 1.0, gen, device)
    rows = [torch.tensor([1.0, 0, 0, 0, 0.62 * e, 0.48 * e, 2 * ez], dtype=torch.float64,
                         device=device)]
    for k in range(3):
        r = (0.03 + 0.06 * u[k, 0]) * e
        rows.append(torch.stack([torch.tensor(7.0, dtype=torch.float64, device=device),
                                 (u[k, 1] - 0.5) * 0.6 * e, (u[k, 2] - 0.5) * 0.45 * e,
                                 (u[k, 3] - 0.5) * 1.4 * ez, r, r, r]))
    return torch.stack(rows)


def _grid(c, device):
    ax = [(torch.arange(n, dtype=torch.float64, device=device) - (n - 1) / 2) * c["voxel"]
          for n in (c["n"], c["n"], c["nz"])]
    return torch.meshgrid(*ax, indexing="ij")


def _spect_inputs(c, seed, device):
    """Object, attenuation map, scatter estimate and Poisson projections of a study."""
    gen = _gen(seed, device)
    ell = _ellipsoids(c, gen, device)
    X, Y, Z = _grid(c, device)
    f = torch.zeros_like(X)
    for a, x, y, z, rx, ry, rz in ell:
        f += a * (((X - x) / rx) ** 2 + ((Y - y) / ry) ** 2 + ((Z - z) / rz) ** 2 <= 1)
    f *= 0.75 + 0.5 * torch.rand(f.shape, generator=gen, device=device, dtype=torch.float64)
    # attenuation: soft tissue with two lungs, slightly textured (cm^-1)
    rx, ry = ell[0, 4], ell[0, 5]
    mu = torch.where((X / rx) ** 2 + (Y / ry) ** 2 <= 1, 0.15, 0.0).double()
    for s in (-1, 1):
        lung = ((X - s * 0.45 * rx) / (0.3 * rx)) ** 2 + (Y / (0.55 * ry)) ** 2 <= 1
        mu = torch.where(lung, 0.04, mu)
    mu = mu * (0.9 + 0.2 * torch.rand(mu.shape, generator=gen, device=device, dtype=torch.float64))
    # expected counts: analytic line integrals (rotating detector), a mean attenuation
    t = (_angles(c).double() * math.pi / 180).to(device)
    y, zz = Y[0, :, 0].view(1, -1, 1), Z[0, 0].view(1, 1, -1)
    lam = torch.zeros((c["angles"], c["n"], c["nz"]), dtype=torch.float64, device=device)
    for a, x0, y0, z0, ex, ey, ez in ell:
        w = torch.sqrt((ex * torch.sin(t)) ** 2 + (ey * torch.cos(t)) ** 2).view(-1, 1, 1)
        u0 = (-x0 * torch.sin(t) + y0 * torch.cos(t)).view(-1, 1, 1)
        q = 1 - ((y - u0) / w) ** 2 - ((zz - z0) / ez) ** 2
        lam += a * 2 * ex * ey / w * torch.sqrt(torch.clamp(q, min=0))
    lam = 0.2 * lam / c["voxel"]
    sc = 0.15 * lam.mean() * torch.ones_like(lam) if c.get("scatter") else None
    counts = torch.poisson((lam if sc is None else lam + sc).float(), generator=gen)
    return f.float(), mu.float(), counts, None if sc is None else sc.float()


def _spect_matrix(c, mu):
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta, SPECTPSFMeta
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTAttenuationTransform, SPECTPSFTransform
    v = c["voxel"]
    om = SPECTObjectMeta([v, v, v], (c["n"], c["n"], c["nz"]))
    pm = SPECTProjMeta((c["n"], c["nz"]), [v, v], [float(a) for a in _angles(c)],
                       radii=_radii(c))
    ts = [SPECTAttenuationTransform(mu)]
    if c["psf"]:
        ts.append(SPECTPSFTransform(SPECTPSFMeta(_PSF)))
    return SPECTSystemMatrix(ts, [], om, pm)


_PSF = (0.03, 0.11)  # sigma(d) = 0.03 d + 0.11 cm


def _prepare_spect(c, seed):
    from pytomography_gb300.likelihoods import PoissonLogLikelihood
    dev = torch.device("cuda", torch.cuda.current_device())
    f, mu, g, s = _spect_inputs(c, seed, dev)
    H = _spect_matrix(c, mu)
    st = {"op": c["op"], "H": H, "subsets": c["subsets"], "sub": None}
    if c["subsets"] > 1:
        H.set_n_subsets(c["subsets"])
        st["sub"] = c["subsets"] // 2
    if c["op"] == "forward":
        st["f"] = f
    elif c["op"] == "backward":
        st["g"] = g if st["sub"] is None else g[st["sub"]::c["subsets"]].contiguous()
    elif c["op"] == "gradient":
        more = [_spect_inputs(c, seed + 7919 * k, dev) for k in range(1, c["batch"])]
        st["f"] = torch.stack([f + 0.1] + [m[0] + 0.1 for m in more])
        st["g"] = torch.stack([g] + [m[2] for m in more])
    else:
        lik = PoissonLogLikelihood(H, g, additive_term=s)
        lik._set_n_subsets(c["subsets"])
        st["lik"] = lik
    return st


def _run_spect(st):
    from pytomography_gb300 import autograd
    from pytomography_gb300.algorithms import BSREM, OSEM
    from pytomography_gb300.priors import RelativeDifferencePrior
    op, H = st["op"], st["H"]
    if op == "forward":
        return H.forward(st["f"], st["sub"])
    if op == "backward":
        return H.backward(st["g"], st["sub"])
    if op == "gradient":
        x = st["f"].requires_grad_(True)
        loss = autograd.poisson_nll(x, H, st["g"])
        return {"loss": loss.detach(), "grad": torch.autograd.grad(loss, x)[0]}
    if op == "osem":
        rec = OSEM(st["lik"])(1, st["subsets"])
        return {"object": rec, "predicted": st["lik"].projections_predicted}
    prior = RelativeDifferencePrior(beta=0.3, gamma=2.0)
    return BSREM(st["lik"], prior=prior)(1, st["subsets"])


# ------------------------------------------------------------------------- serving
def _studies(c):
    out = []
    for item in c["mix"].split(","):
        n, a = (int(v) for v in item.split("x"))
        out.append({"n": n, "nz": n, "angles": a, "subsets": c["subsets"], "psf": True,
                    "voxel": c["voxel"], "radius": c["radius"], "orbit": 0.0, "scatter": False})
    return out


def _prepare_serving(c, seed):
    from pytomography_gb300.batched import BatchedOSEM
    from pytomography_gb300.likelihoods import PoissonLogLikelihood
    dev = torch.device("cuda", torch.cuda.current_device())
    liks = []
    for k, s in enumerate(_studies(c)):
        _, mu, g, _ = _spect_inputs(s, seed + 7919 * k, dev)
        liks.append(PoissonLogLikelihood(_spect_matrix(s, mu), g))
    return {"batch": BatchedOSEM(liks, n_subsets=c["subsets"])}


# ------------------------------------------------------------------------- PET inputs
def _scanner(c):
    """Crystal ring geometry in the form the metadata classes take."""
    return dict(crystalTransNr=1, crystalTransSpacing=4.0, submoduleTransNr=1,
                submoduleTransSpacing=0.0, moduleTransNr=1, moduleTransSpacing=0.0,
                rsectorTransNr=c["crystals"], crystalAxialNr=c["rings"], crystalAxialSpacing=4.0,
                submoduleAxialNr=1, submoduleAxialSpacing=0.0, moduleAxialNr=1,
                moduleAxialSpacing=0.0, rsectorAxialNr=1, radius=400.0, firstCrystalAxis=1,
                NrCrystalsPerRing=c["crystals"], NrRings=c["rings"], min_rsector_difference=0)


_TOF_RANGE, _TOF_FWHM = 650.0, 58.5  # mm


def _pet_image(c, gen, device):
    n, v = (c["nx"], c["nx"], c["nz"]), c["voxel"]
    ax = [(torch.arange(k, dtype=torch.float64, device=device) - (k - 1) / 2) * v for k in n]
    X, Y, Z = torch.meshgrid(*ax, indexing="ij")
    e, ez = n[0] * v / 2, n[2] * v / 2
    f = ((X / (0.75 * e)) ** 2 + (Y / (0.5 * e)) ** 2 <= 1).double()
    u = _uniform((2, 3), -0.5, 0.5, gen, device)
    for k in range(2):
        d2 = (X - u[k, 0] * e) ** 2 + (Y - u[k, 1] * 0.7 * e) ** 2 + (Z - u[k, 2] * ez) ** 2
        f += 3.0 * (d2 <= (0.12 * e) ** 2)
    f *= 0.75 + 0.5 * torch.rand(f.shape, generator=gen, device=device, dtype=torch.float64)
    return f.float()


def _pet_events(c, gen, device):
    """Listmode events [E, 2 or 3]: emission points in an ellipsoid with isotropic directions
    that hit the scanner, a TOF bin around the emission point, and 20% uniform randoms."""
    E, R, nt, nr = c["events"], 400.0, c["crystals"], c["rings"]
    zh = (nr - 1) * 4.0 / 2
    n_true, chunks, got = E - E // 5, [], 0
    zr = min(80.0, 0.8 * zh)
    while got < n_true:
        m = 3 * (n_true - got) + 1000
        p = _uniform((m, 3), -1, 1, gen, device)
        p = p[(p * p).sum(1) <= 1] * torch.tensor([150.0, 100.0, zr], dtype=torch.float64,
                                                  device=device)
        u = torch.randn((len(p), 3), generator=gen, device=device, dtype=torch.float64)
        u = u / u.norm(dim=1, keepdim=True)
        a = u[:, 0] ** 2 + u[:, 1] ** 2
        b = 2 * (p[:, 0] * u[:, 0] + p[:, 1] * u[:, 1])
        d = torch.sqrt(torch.clamp(b * b - 4 * a * (p[:, 0] ** 2 + p[:, 1] ** 2 - R * R), min=0))
        q1 = p + ((-b - d) / (2 * a + 1e-30))[:, None] * u
        q2 = p + ((-b + d) / (2 * a + 1e-30))[:, None] * u
        ok = (q1[:, 2].abs() <= zh) & (q2[:, 2].abs() <= zh) & (a > 1e-6)
        p, q1, q2 = p[ok], q1[ok], q2[ok]
        ids = []
        for q in (q1, q2):
            tr = torch.round(torch.atan2(q[:, 1], q[:, 0]) / (2 * math.pi / nt)).long() % nt
            ring = torch.clamp(torch.round((zh - q[:, 2]) / 4.0).long(), 0, nr - 1)
            ids.append(ring * nt + tr)
        cols = ids
        if c["bins"]:
            w = q2 - q1
            s = ((p - (q1 + q2) / 2) * w).sum(1) / w.norm(dim=1)
            s = s + _TOF_FWHM / 2.355 * torch.randn(len(s), generator=gen, device=device,
                                                    dtype=torch.float64)
            tb = torch.round(s / (_TOF_RANGE / c["bins"])).long() + (c["bins"] - 1) // 2
            cols = ids + [torch.clamp(tb, 0, c["bins"] - 1)]
        ev = torch.stack(cols, 1)[ids[0] != ids[1]]
        chunks.append(ev)
        got += len(ev)
    rnd = lambda hi: torch.randint(0, hi, (E // 5,), generator=gen, device=device)  # noqa: E731
    i = rnd(nt * nr)
    j = rnd(nt * nr - 1)
    cols = [i, j + (j >= i)] + ([rnd(c["bins"])] if c["bins"] else [])
    ev = torch.cat([torch.cat(chunks)[:n_true], torch.stack(cols, 1)])
    return ev[torch.randperm(len(ev), generator=gen, device=device)].cpu()


def _sensitivity_pairs(c, gen, device):
    """A sample of 400k crystal pairs for the sensitivity image."""
    n = c["crystals"] * c["rings"]
    i = torch.randint(0, n, (400_000,), generator=gen, device=device)
    j = torch.randint(0, n - 1, (400_000,), generator=gen, device=device)
    return torch.stack([i, j + (j >= i)], 1).cpu()


def _pet_inputs(c, seed, device):
    gen = _gen(seed, device)
    out = {"img": _pet_image(c, gen, device)}
    if c["path"] == "pet_lm":
        out["events"] = _pet_events(c, gen, device)
        out["pairs"] = _sensitivity_pairs(c, gen, device) if c["op"] == "osem" else None
        out["w"] = (0.5 + torch.rand(c["events"], generator=gen, device=device)).float()
        return out
    n_sel = len(range(c["subsets"] // 2, c["crystals"] // 2, c["subsets"]))
    shape = [n_sel, c["crystals"] + 1, c["rings"] ** 2] + ([c["bins"]] if c["bins"] else [])
    if c["op"] == "backward":
        lam = torch.full(shape, 2.0, device=device)
        out["sino"] = torch.poisson(lam, generator=gen)
    return out


_ADDITIVE = 0.05  # expected randoms of an event's LOR and TOF bin


def _prepare_pet(c, seed):
    from pytomography_gb300.likelihoods import PoissonLogLikelihood
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import (PETLMProjMeta, PETSinogramPolygonProjMeta,
                                                 PETTOFMeta)
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix, PETSinogramSystemMatrix
    dev = torch.device("cuda", torch.cuda.current_device())
    x = _pet_inputs(c, seed, dev)
    om = ObjectMeta([c["voxel"]] * 3, (c["nx"], c["nx"], c["nz"]))
    tof = PETTOFMeta(c["bins"], _TOF_RANGE, _TOF_FWHM) if c["bins"] else None
    st = {"op": c["op"], "subsets": c["subsets"], "sub": c["subsets"] // 2, "f": x["img"]}
    if c["path"] == "pet_sino":
        H = PETSinogramSystemMatrix(om, PETSinogramPolygonProjMeta(_scanner(c), tof),
                                    device=str(dev))
        st["p"] = x.get("sino")
    else:
        pm = PETLMProjMeta(x["events"], info=_scanner(c), tof_meta=tof,
                           detector_ids_sensitivity=x["pairs"])
        H = PETLMSystemMatrix(om, pm, compute_sensitivity=c["op"] == "osem")
    H.set_n_subsets(c["subsets"])
    st["H"] = H
    if c["op"] == "backward" and c["path"] == "pet_lm":
        st["p"] = x["w"][st["sub"]::c["subsets"]].contiguous()
    if c["op"] == "osem":
        add = torch.full((c["events"],), _ADDITIVE, device=dev)
        st["lik"] = PoissonLogLikelihood(H, additive_term=add)
        st["lik"]._set_n_subsets(c["subsets"])
    return st


def _run_pet(st):
    from pytomography_gb300.algorithms import OSEM
    if st["op"] == "forward":
        return st["H"].forward(st["f"], st["sub"])
    if st["op"] == "backward":
        return st["H"].backward(st["p"], st["sub"])
    return OSEM(st["lik"])(1, st["subsets"])


# ------------------------------------------------------------------------- entry points
def prepare(case, seed):
    if case["path"] == "spect":
        return {"run": _run_spect, **_prepare_spect(case, seed)}
    if case["path"] == "serving":
        return {"run": lambda st: st["batch"](1), **_prepare_serving(case, seed)}
    return {"run": _run_pet, **_prepare_pet(case, seed)}


def run(state):
    return state["run"](state)


def _pad_size(n):
    return int(math.ceil((math.sqrt(2) * n - n) / 2))


def _sigma(c, radius, n_pad):
    k = torch.arange(n_pad, dtype=torch.float64)
    d = (n_pad / 2 - k - 0.5) if n_pad % 2 == 0 else ((n_pad - 1) / 2 - k)
    return _PSF[0] * torch.clamp(radius + d * c["voxel"], min=0) + _PSF[1]


def _spect_work(c, passes):
    """``passes``: projections of one angle, forward or back, per listed angle."""
    vox, q = c["n"] * c["n"] * c["nz"], c["n"] * c["nz"]
    flops = 8.0  # a bilinear sample and the attenuation product
    if c["psf"]:
        L = c["n"] + 2 * _pad_size(c["n"])
        s = _sigma(c, c["radius"], L) / c["voxel"]
        half = torch.minimum(torch.ceil(5.7 * s), torch.ceil(3 * s.max()))
        flops += 4.0 * float((2 * half + 1).mean())  # y and z taps, a multiply-add each
    return passes * vox * flops, 4 * vox, 4 * q


def work(case):
    c = case
    if c["path"] == "serving":
        tot = {"bytes": 0.0, "flops": 0.0}
        for s in _studies(c):
            fl, vox, q = _spect_work(s, 2 * s["angles"])
            tot["flops"] += fl
            tot["bytes"] += s["subsets"] * 5 * vox + 2 * s["angles"] * q
        return tot
    if c["path"] == "spect":
        n_sel = len(range(c["subsets"] // 2 if c["subsets"] > 1 else 0, c["angles"], c["subsets"]))
        if c["op"] in ("forward", "backward"):  # object and attenuation map, projections
            fl, vox, q = _spect_work(c, n_sel)
            return {"bytes": 2 * vox + n_sel * q, "flops": fl}
        fl, vox, q = _spect_work(c, 2 * c["angles"] * c["batch"])
        if c["op"] == "gradient":  # object in, gradient out, counts in
            return {"bytes": c["batch"] * (2 * vox + c["angles"] * q) + vox, "flops": fl}
        # a sub-iteration reads the object, the map and the normalisation and writes the object
        more = 1 if c["op"] == "bsrem" else 0
        add = 1 if c["scatter"] else 0
        flops = fl + (c["subsets"] * c["n"] ** 2 * c["nz"] * 26 * 10.0 if more else 0.0)
        return {"bytes": c["subsets"] * (4 + more) * vox + (1 + add) * c["angles"] * q,
                "flops": flops}
    vox = 4 * c["nx"] * c["nx"] * c["nz"]
    if c["path"] == "pet_lm":
        n = len(range(c["subsets"] // 2, c["events"], c["subsets"]))
        # planes of a LOR inside the image and, with TOF, inside the 3-sigma window
        planes = 0.65 * c["nx"]
        if c["bins"]:
            planes = min(planes, (6 * _TOF_FWHM / 2.355 + _TOF_RANGE / c["bins"]) / c["voxel"])
        flops = 12.0 * planes
        if c["op"] == "osem":
            return {"bytes": c["subsets"] * 3 * vox + c["events"] * 20.0,
                    "flops": 2 * c["events"] * flops}
        return {"bytes": vox + n * 16.0, "flops": n * flops}
    n_ang = len(range(c["subsets"] // 2, c["crystals"] // 2, c["subsets"]))
    n = n_ang * (c["crystals"] + 1) * c["rings"] ** 2 * max(1, c["bins"])
    planes = 0.65 * c["nx"]
    if c["bins"]:
        planes = min(planes, (6 * _TOF_FWHM / 2.355 + _TOF_RANGE / c["bins"]) / c["voxel"])
    return {"bytes": vox + n * 4.0, "flops": n * 12.0 * 0.6 * planes}


# ------------------------------------------------------------------- 64-bit restatement
def _rotate(x, deg):
    """[H, H, Z] rotated about its centre by ``deg`` (bilinear, zeros outside)."""
    a = deg * math.pi / 180
    th = torch.tensor([[[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0]]],
                      dtype=torch.float64, device=x.device)
    img = x.permute(2, 0, 1).unsqueeze(0)
    grid = F.affine_grid(th, list(img.shape), align_corners=True)
    r = F.grid_sample(img, grid, mode="bilinear", padding_mode="zeros", align_corners=True)
    return r[0].permute(1, 2, 0)


class _Exact:
    """Rotate, attenuate, blur and sum, one angle at a time."""

    def __init__(self, c, mu):
        self.c, self.pad = c, _pad_size(c["n"])
        self.L = c["n"] + 2 * self.pad
        self.mu = self._padded(mu.double())
        self.angles = [float(a) for a in _angles(c)]
        self.radii = _radii(c)
        self.taps = {}
        if c["psf"]:
            for r in set(self.radii):
                s = _sigma(c, r, self.L) / c["voxel"]
                h = int(math.ceil(float(s.max()) * 3))
                x = torch.arange(-h, h + 1, dtype=torch.float64)
                k = torch.exp(-x[None] ** 2 / (2 * s[:, None] ** 2 + DELTA))
                self.taps[r] = (k / k.sum(1, keepdim=True)).to(mu.device)

    def _padded(self, x):
        p = self.pad
        return F.pad(x, [0, 0, p, p, p, p])

    def _attenuation(self, beta):
        v = _rotate(self.mu, beta - 270.0) * self.c["voxel"]
        rev = torch.flip(torch.cumsum(torch.flip(v, (0,)), 0), (0,))
        return torch.exp(-(rev - v / 2))

    def _blur(self, x, a):
        if not self.taps:
            return x
        w = self.taps[self.radii[a]]
        h = w.shape[1] // 2
        for dim in (1, 2):
            n = x.shape[dim]
            xp = F.pad(x, [0, 0, h, h] if dim == 1 else [h, h])
            y = torch.zeros_like(x)
            for t in range(2 * h + 1):
                y = y + w[:, t].view(-1, 1, 1) * xp.narrow(dim, t, n)
            x = y
        return x

    def forward(self, f, a):
        b = self.angles[a]
        v = _rotate(self._padded(f), b - 270.0) * self._attenuation(b)
        return self._blur(v, a).sum(0)[self.pad:self.pad + self.c["n"]]

    def backward(self, g, a):
        b, p, n = self.angles[a], self.pad, self.c["n"]
        v = F.pad(g, [0, 0, p, p]).unsqueeze(0).expand(self.L, -1, -1)
        v = self._blur(v, a) * self._attenuation(b)
        return _rotate(v, 270.0 - b)[p:p + n, p:p + n]

    def back(self, g, idx):
        return sum(self.backward(g[k], a) for k, a in enumerate(idx))


def _rdp_gradient(f, beta, gamma):
    """Gradient of the relative-difference prior, isotropic voxels, replicated edges."""
    p = F.pad(f[None, None], (1,) * 6, mode="replicate")[0, 0]
    nx, ny, nz = f.shape
    out = torch.zeros_like(f)
    for i in (0, 1, 2):
        for j in (0, 1, 2):
            for k in (0, 1, 2):
                if i == j == k == 1:
                    continue
                w = 1 / math.sqrt((i - 1) ** 2 + (j - 1) ** 2 + (k - 1) ** 2)
                s = p[i:i + nx, j:j + ny, k:k + nz]
                d = f - s
                num = d * (gamma * d.abs() + 3 * s + f + 2 * DELTA)
                out += w * num / (f + s + gamma * d.abs() + DELTA) ** 2
    return beta * out


def _exact_em(c, inputs, kind):
    """One iteration of OSEM, or of BSREM with the relative-difference prior, from ones."""
    _, mu, g, s = inputs
    P, m, g = _Exact(c, mu), c["subsets"], g.double()
    s = None if s is None else s.double()
    f = torch.ones((c["n"], c["n"], c["nz"]), dtype=torch.float64, device=mu.device)
    subs = [list(range(k, c["angles"], m)) for k in range(m)]
    ones = torch.ones_like(g[0])
    norm = [sum(P.backward(ones, a) for a in idx) for idx in subs]
    total = sum(norm)
    for k, idx in enumerate(subs):
        pred = torch.stack([P.forward(f, a) for a in idx])
        if s is not None:
            pred = pred + s[idx]
        grad = P.back(g[idx] / (pred + DELTA), idx) - norm[k]
        if kind == "osem":
            f = torch.clamp(f + f / (norm[k] + DELTA) * grad, min=0)
        else:
            w = len(idx) / c["angles"]
            grad = grad - w * _rdp_gradient(f, 0.3, 2.0)
            f = torch.clamp(f + f / (w * total + DELTA) * grad, min=1e-4)
    return f, pred


def _exact_spect(c, seed, dev):
    inputs = _spect_inputs(c, seed, dev)
    f, mu, g, _ = inputs
    sub = c["subsets"] // 2 if c["subsets"] > 1 else 0
    idx = list(range(sub, c["angles"], c["subsets"]))
    if c["op"] in ("forward", "backward"):
        P = _Exact(c, mu)
        if c["op"] == "forward":
            return torch.stack([P.forward(f.double(), a) for a in idx])
        return P.back(g[idx].double(), idx)
    if c["op"] == "gradient":
        P, grads = _Exact(c, mu), []
        for b in range(c["batch"]):
            fb, _, gb, _ = _spect_inputs(c, seed + 7919 * b, dev)
            x = (fb + 0.1).double().requires_grad_(True)
            acc = torch.zeros_like(x)
            for a in idx:
                pred = P.forward(x, a)
                nll = (pred - gb[a].double() * torch.log(pred + DELTA)).sum()
                acc += torch.autograd.grad(nll, x)[0]
            grads.append(acc)
        # the loss is a sum with cancellation: no value is given for its last digits
        return {"loss": None, "grad": torch.stack(grads)}
    rec, pred = _exact_em(c, inputs, c["op"])
    return {"object": rec, "predicted": pred} if c["op"] == "osem" else rec


def _lut(c):
    """Crystal centres [n, 3] (mm, single precision as the scanner files give them)."""
    t = torch.arange(c["crystals"]) / c["crystals"] * 2 * math.pi
    z = torch.arange(c["rings"]) * 4.0 - (c["rings"] - 1) * 4.0 / 2
    xy = 400.0 * torch.stack([torch.cos(t), torch.sin(t)], 1)
    return torch.cat([xy.repeat(c["rings"], 1), -z.repeat_interleave(c["crystals"])[:, None]], 1)


class _Joseph:
    """Joseph line integrals between end points p0, p1 [E, 3], optionally TOF weighted
    (``bins``: the bin index counted from the central one)."""

    def __init__(self, c, p0, p1, bins=None):
        self.n = (c["nx"], c["nx"], c["nz"])
        self.v = float(torch.tensor(c["voxel"], dtype=torch.float32))
        self.org = [(-k / 2 + 0.5) * c["voxel"] for k in self.n]
        self.p0, self.d = p0, p1 - p0
        self.len = self.d.norm(dim=1)
        self.bins = bins
        if bins is not None:
            edges = torch.linspace(-1, 1, c["bins"] + 1) * _TOF_RANGE / 2
            self.bw = float(edges[1] - edges[0])
            self.sig = float(torch.tensor(_TOF_FWHM / 2.355, dtype=torch.float32))
            self.off = -self.bw / 2 if c["bins"] % 2 == 0 else 0.0

    def _axis(self):
        ad = self.d.abs()
        k = torch.zeros(len(ad), dtype=torch.long, device=ad.device)
        k[ad[:, 1] > ad[:, 0]] = 1
        k[ad[:, 2] > torch.maximum(ad[:, 0], ad[:, 1])] = 2
        return k

    def _steps(self):
        """(events, flat voxel index, weight) of every plane and corner."""
        axis = self._axis()
        strides = (self.n[1] * self.n[2], self.n[2], 1)
        for k in range(3):
            ev = torch.where((axis == k) & (self.len > 0))[0]
            if not len(ev):
                continue
            a, b = (k + 1) % 3, (k + 2) % 3
            p0, d, ln = self.p0[ev], self.d[ev], self.len[ev]
            cf = self.v * ln / d[:, k].abs()
            lo = torch.minimum(p0[:, k], p0[:, k] + d[:, k])
            hi = torch.maximum(p0[:, k], p0[:, k] + d[:, k])
            for i in range(self.n[k]):
                x = self.org[k] + i * self.v
                t = (x - p0[:, k]) / d[:, k]
                w = cf * ((x >= lo) & (x <= hi))
                if self.bins is not None:
                    s = ((t - 0.5) * ln - (self.bins[ev] * self.bw + self.off)).abs()
                    q = 1 / (math.sqrt(2) * self.sig)
                    tw = 0.5 * (torch.erfc((s - self.bw / 2) * q) -
                                torch.erfc((s + self.bw / 2) * q))
                    w = w * tw * (s <= 3 * self.sig + self.bw / 2)
                fa = (p0[:, a] + t * d[:, a] - self.org[a]) / self.v
                fb = (p0[:, b] + t * d[:, b] - self.org[b]) / self.v
                ia, ib = torch.floor(fa), torch.floor(fb)
                for qa in (0, 1):
                    for qb in (0, 1):
                        ja, jb = ia + qa, ib + qb
                        ok = (ja >= 0) & (ja < self.n[a]) & (jb >= 0) & (jb < self.n[b]) & (w > 0)
                        wq = (fa - ia if qa else 1 - fa + ia) * (fb - ib if qb else 1 - fb + ib)
                        at = i * strides[k] + ja * strides[a] + jb * strides[b]
                        yield ev, torch.where(ok, at, 0).long(), torch.where(ok, w * wq, 0)

    def forward(self, img):
        out, flat = torch.zeros(len(self.d), dtype=torch.float64, device=img.device), img.reshape(-1)
        for ev, at, w in self._steps():
            out[ev] += w * flat[at]
        return out

    def backward(self, p):
        out = torch.zeros(self.n, dtype=torch.float64, device=p.device)
        for ev, at, w in self._steps():
            out.view(-1).index_add_(0, at, w * p[ev])
        return out


def _sino_lors(c, angles):
    """End points [E, 3] twice of the sinogram elements (angle, radial, ring pair): crystal
    ids counted from half a crystal on, ring pairs by increasing ring difference; a bin that
    no crystal pair reaches keeps (0, 0)."""
    n, nr, lut = c["crystals"], c["rings"], _lut(c)
    k1, k2 = torch.tril_indices(n, n)  # crystal 1 >= crystal 2
    a, b = ((k.double() - 0.5) % n for k in (k1, k2))
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    s = lo + hi
    outer = (s >= 1.5 * n) | (s < 0.5 * n)
    r = torch.where(outer, hi - lo - n / 2, n / 2 - (hi - lo))
    r = torch.floor(torch.where(lo == hi, torch.where(outer, -n / 2, n / 2).double(), r))
    ang = torch.where(s < n / 2, (2 * lo + n + r) / 2,
                      torch.where(s >= 1.5 * n, (2 * lo - n + r) / 2, (2 * lo - r) / 2))
    ang, rad = torch.floor(ang).long(), torch.floor(r + (n + 1) / 2).long()
    det = torch.zeros((n // 2, n + 1, 4))
    flat = ang * (n + 1) + rad
    last = torch.full((n // 2 * (n + 1),), -1).scatter_reduce(
        0, flat, torch.arange(len(flat)), "amax")  # the last pair in id order keeps the bin
    at = last[last >= 0]
    det.view(-1, 4)[last >= 0] = torch.cat([lut[k1[at], :2], lut[k2[at], :2]], 1)
    rings = [(i, i) for i in range(nr)]
    for diff in range(1, nr):
        rings += [(i, i + diff) for i in range(nr - diff)]
        rings += [(i + diff, i) for i in range(nr - diff)]
    z = lut[torch.tensor(rings) * n, 2]  # [P, 2]
    d = det[angles]
    shape = (*d.shape[:2], len(rings))
    pts = []
    for k in (0, 1):
        xy = d[:, :, None, 2 * k:2 * k + 2].expand(*shape, 2)
        pts.append(torch.cat([xy, z[:, k].expand(shape)[..., None]], -1).reshape(-1, 3))
    return pts


def _exact_sino(c, x, dev):
    idx = list(range(c["subsets"] // 2, c["crystals"] // 2, c["subsets"]))
    p0, p1 = (p.double().to(dev) for p in _sino_lors(c, idx))
    nb = c["bins"]
    img = torch.zeros((c["nx"], c["nx"], c["nz"]), dtype=torch.float64, device=dev)
    cols = []
    for b in range(max(1, nb)):
        tb = torch.full((len(p0),), b - (nb - 1) // 2, device=dev) if nb else None
        J = _Joseph(c, p0, p1, tb)
        if c["op"] == "forward":
            cols.append(J.forward(x["img"].double()))
        else:
            p = x["sino"].double()
            img += J.backward((p[..., b] if nb else p).reshape(-1))
    if c["op"] == "backward":
        return img
    out = torch.stack(cols, 1) if nb else cols[0]
    return out.reshape(len(idx), c["crystals"] + 1, c["rings"] ** 2, *([nb] if nb else [])).squeeze()


def _exact_pet(c, seed, dev):
    x = _pet_inputs(c, seed, dev)
    sub, m = c["subsets"] // 2, c["subsets"]
    if c["path"] == "pet_sino":
        return _exact_sino(c, x, dev)
    lut = _lut(c).double().to(dev)

    def lors(k):
        e = x["events"][k::m].to(dev)
        return _Joseph(c, lut[e[:, 0]], lut[e[:, 1]],
                       e[:, 2] - (c["bins"] - 1) // 2 if c["bins"] else None)

    if c["op"] == "forward":
        return lors(sub).forward(x["img"].double())
    if c["op"] == "backward":
        return lors(sub).backward(x["w"][sub::m].double())
    pairs = x["pairs"].to(dev)
    sens = _Joseph(c, lut[pairs[:, 0]], lut[pairs[:, 1]]).backward(
        torch.full((len(pairs),), 1 + DELTA, dtype=torch.float64, device=dev))
    sens[sens < 1e-7] = 1e7
    f = torch.ones(sens.shape, dtype=torch.float64, device=dev)
    z = (c["nz"] - 1) / 2 + torch.stack([lut[:, 2].min(), lut[:, 2].max()]) / c["voxel"]
    f[:, :, :max(0, math.ceil(float(z[0])))] = 0
    f[:, :, max(0, math.floor(float(z[1]))):] = 0
    for k in range(m):
        J = lors(k)
        frac = len(J.d) / c["events"]
        bp = J.backward(1 / (J.forward(f) + _ADDITIVE + DELTA))
        f = torch.clamp(f + f / (frac * sens + DELTA) * (bp - frac * sens), min=0)
    return f


def exact(case, seed):
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    if case["path"] == "spect":
        return _exact_spect(case, seed, dev)
    if case["path"] == "serving":
        out = []
        for k, s in enumerate(_studies(case)):
            out.append(_exact_em(s, _spect_inputs(s, seed + 7919 * k, dev), "osem")[0])
        return out
    return _exact_pet(case, seed, dev)
