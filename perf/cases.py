"""The calls whose speed matters to a user of this framework, as cases that can be timed and checked.

A refinement driver (PSO, simplex, grid or pattern search) holds one job and scores candidate poses, one at a
time or a generation at a time; the stages of that call are also public entry points of their own (density,
templates, particle preparation, correlation), and two more paths surround the search: the preparation of a raw
particle stack and the geometric restraint of a pose. Each kind of case below is one of those calls:

  score        ScoringJob.score, one pose (blocks until the score is on the host, as a simplex step needs it)
  generation   BatchScoringJob.score_batch, one generation of poses, in the precision the caller chooses
  templates    IntegratedProjector.build_templates, one density, many directions
  particles    ParticleFourierPreparer.prepare_batch, a stack of particles at its in-plane angles
  correlate    correlate_templates_and_particle, the reference's per-particle call
  density      MovedChainDensity.generate, one pose of the moving chain on its fixed context
  ingest       ingest.preprocess_stack, shift, crop, whitening and high-pass of a raw stack
  restraint    GeometryRestraint.evaluate_many, overlap and separation of a list of poses

Inputs have the published shapes: box 64 / 200 particles, box 128 / 5,000 particles and box 256 of the workloads
in gisapr_gb300/synthetic.py, with the serving stream's boxes 96 and 192. Particles are projections of the model
under a CTF at a signal-to-noise ratio of 0.05 and normalised; densities handed to the projector directly are
blobs with noise in every shell, as a measured map has.

``score`` and ``generation`` return what a driver and the search text are made from in floating point: the scores
and every particle's peak and z-score. (The place of a maximum is left to ``correlate``: over tens of thousands of
maps two places can be equal to the last bit of float32.) A generation's scores are sums in 64 bits over float32
peaks and are returned as float32.
"""
import math
import os
import tempfile

import numpy as np
import torch

DEV = "cuda:0"
# box -> (A per pixel, HEALPix order, local range, psi step, crop, half-maximum resolution of the FSC or None)
SEARCH = {64: (1.5, 2, 15.0, 15.0, 10, None), 96: (1.1, 3, 10.0, 7.5, 12, 4.0), 128: (1.1, 3, 10.0, 7.5, 12, 4.0),
          192: (1.1, 3, 10.0, 7.5, 12, 4.0), 256: (0.85, 4, 6.0, 3.75, 14, 4.0)}


def listed():
    return [
        # one simplex step of a small job (the box-64 workload): a dozen short launches, latency is all of it
        dict(name="score_box64_200p", kind="score", box=64, particles=200, moving=760, fixed=3030),
        # one simplex step of the headline workload: box 128, 5,000 particles, 3,000 + 20,000 atoms
        dict(name="score_box128_5kp", kind="score", box=128, particles=5000, moving=3000, fixed=20000),
        # one PSO generation of 64 poses with the split tensor-core correlation, the form a batch user picks
        dict(name="gen64_box128_fp16x3", kind="generation", box=128, particles=2000, moving=3000, fixed=20000,
             poses=64, precision="fp16x3"),
        # a small swarm on a small job in plain float32
        dict(name="gen24_box64_fp32", kind="generation", box=64, particles=200, moving=760, fixed=3030, poses=24,
             precision="fp32"),
        # the template bank of one density at the headline box: every HEALPix order-3 direction
        dict(name="templates_box128_768", kind="templates", box=128, newbox=128, dirs=768, masked=True),
        # the same at a box that is not a power of two (the serving stream's 192)
        dict(name="templates_box192_500", kind="templates", box=192, newbox=192, dirs=500, masked=True),
        # the largest box: box 256, a third of the HEALPix order-4 directions
        dict(name="templates_box256_1000", kind="templates", box=256, newbox=256, dirs=1000, masked=True),
        # loading a job: 2,000 particles at their three in-plane angles
        dict(name="particles_box128_2k", kind="particles", box=128, newbox=128, n=2000, psi=3, masked=True),
        # the reference's per-particle call: a handful of local directions against one particle
        dict(name="correlate_box128_6x3", kind="correlate", box=128, crop=12, dirs=6, psi=3),
        # one density of a moved 3,000-atom chain
        dict(name="density_box128", kind="density", box=128, apix=1.1, moving=3000, fixed=20000),
        # raw 256-pixel particles cropped to 128, whitened and high-passed
        dict(name="ingest_256_to_128", kind="ingest", size=256, crop=128, n=500, whitening=True, highpass=True),
        # the restraint of one swarm against the main body, at the command's default box and pixel size
        dict(name="restraint_box256_16", kind="restraint", box=256, apix=1.5, moving=3000, fixed=20000, poses=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score", "generation", "templates", "particles", "correlate", "density", "ingest",
                       "restraint"])
    if kind in ("score", "generation"):
        c = dict(kind=kind, box=rng.choice([64, 96, 128] if kind == "score" else [64, 96, 128, 128]),
                 particles=_log(rng, 100, 4000 if kind == "score" else 800), moving=_log(rng, 200, 3000),
                 fixed=_log(rng, 600, 20000))
        if kind == "generation":
            c.update(poses=rng.randint(5, 48), precision=rng.choice(["fp32", "fp16x3", "fp16", "bf16x3"]))
        return c
    if kind == "templates":
        box = rng.choice([32, 64, 96, 128, 128, 192, 256])
        return dict(kind=kind, box=box, newbox=box if rng.random() < 0.75 else 16 * max(2, box // 32),
                    dirs=_log(rng, 5, 800 if box >= 192 else 2000), masked=rng.random() < 0.8)
    if kind == "particles":
        box = rng.choice([64, 96, 128, 128, 192, 256])
        return dict(kind=kind, box=box, newbox=box if rng.random() < 0.75 else 16 * (box // 32),
                    n=_log(rng, 20, 1500 * 128 * 128 // (box * box)), psi=rng.choice([1, 3, 3, 5]),
                    masked=rng.random() < 0.8)
    if kind == "correlate":
        return dict(kind=kind, box=rng.choice([64, 96, 128, 192, 256]), crop=rng.choice([8, 10, 12, 14]),
                    dirs=_log(rng, 1, 60), psi=rng.choice([1, 3, 5, 7]))
    if kind == "density":
        return dict(kind=kind, box=rng.choice([48, 64, 90, 96, 128, 147, 192, 256]),
                    apix=round(rng.uniform(0.85, 1.6), 2), moving=_log(rng, 150, 8000), fixed=_log(rng, 600, 20000))
    if kind == "ingest":
        size = rng.choice([96, 151, 192, 256])
        return dict(kind=kind, size=size, crop=rng.choice([0, 64, 91]), n=_log(rng, 10, 300),
                    whitening=rng.random() < 0.8, highpass=rng.random() < 0.5)
    return dict(kind=kind, box=rng.choice([96, 150, 200, 256]), apix=round(rng.uniform(1.2, 2.0), 2),
                moving=_log(rng, 200, 3000), fixed=_log(rng, 2000, 20000), poses=rng.randint(1, 16))


# ----------------------------------------------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _euler(rot, tilt, psi):
    """Rows of the Euler frame (RELION's ZYZ), [n, 3, 3] float64."""
    a, b, g = (torch.deg2rad(v) for v in (rot, tilt, psi))
    ca, sa, cb, sb, cg, sg = a.cos(), a.sin(), b.cos(), b.sin(), g.cos(), g.sin()
    return torch.stack([cg * cb * ca - sg * sa, cg * cb * sa + sg * ca, -cg * sb,
                        -sg * cb * ca - cg * sa, -sg * cb * sa + cg * ca, sg * sb,
                        sb * ca, sb * sa, cb], -1).reshape(*a.shape, 3, 3)


def _directions(n, g):
    """n uniform directions as (rot, tilt) degrees, float64 on the device."""
    u = torch.rand(2, n, generator=g, device=DEV, dtype=torch.float64)
    return u[0] * 360 - 180, torch.rad2deg(torch.acos(2 * u[1] - 1))


def _soft_mask(n, radius, edge=6):
    i = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
    d = (i[:, None] ** 2 + i[None] ** 2).sqrt()
    rim = 0.5 * (1 + torch.cos(math.pi * (d - radius) / edge))
    return torch.where(d <= radius, 1.0, torch.where(d <= radius + edge, rim, 0.0))


def _fsc(box, apix, half_res):
    """Shell values of a logistic FSC (ones without a half-maximum resolution)."""
    if half_res is None:
        return np.ones(box, np.float32)
    freq = np.arange(box) / (box * apix)
    return (1.0 / (1.0 + np.exp((freq * half_res - 1.0) / 0.08))).astype(np.float32)


def _packed_fsc(values, n):
    """Shell values on the packed half plane (rows and columns in transform order), float32 values as float64."""
    i = torch.arange(n, device=DEV) - n // 2
    shell = (i[:, None] ** 2 + i[None] ** 2).double().sqrt().long()
    v = torch.as_tensor(values, device=DEV).double()
    full = torch.where(shell < len(v), v[shell.clamp(max=len(v) - 1)], 0.0)
    return torch.fft.ifftshift(full)[:, : n // 2 + 1].contiguous()


def _ctf(n, apix, dfu, dfv, dfa, kk=3.0, voltage=300.0, cs=2.7):
    """CTF times the ISSPA weight on the packed half plane, [particles, n, n/2+1] float64, and the bare CTF."""
    kv = voltage * 1e3
    lam = 12.2643247 / math.sqrt(kv * (1 + kv * 0.978466e-6))
    fy = (torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) / apix)[:, None]
    fx = (torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64) / (n * apix))[None]
    fx = torch.where(fx == 0.5 / apix, -fx, fx)  # the packed plane's last column is the negative Nyquist one
    u2 = fx * fx + fy * fy
    a = torch.deg2rad(dfa)[:, None, None]
    u, v = dfu[:, None, None], dfv[:, None, None]
    s, c = a.sin(), a.cos()
    t = (-u * c * c - v * s * s) * fx * fx + 2 * (-u * s * c + v * s * c) * fx * fy + (-u * s * s - v * c * c) * fy * fy
    gamma = math.pi * lam * t + math.pi / 2 * cs * 1e7 * lam ** 3 * u2 * u2 - math.atan(0.1 / math.sqrt(0.99))
    ctf = -torch.sin(gamma)
    signal = torch.exp(-78.7757 * u2 - 12.9121 * u2.sqrt() + 1.28732) / (kk + 1)
    noise = torch.exp(-9.32 * u2 + 2.65 * u2.sqrt() + 0.01908) / signal
    return ctf / (noise + kk * ctf * ctf).sqrt(), ctf


def _defocus(n, g):
    u = torch.rand(3, n, generator=g, device=DEV, dtype=torch.float64)
    dfu = (1e4 + 1.5e4 * u[0]).float()
    return dfu, (dfu + (3000 * u[1] - 1500).float()).clamp(1e4, 2.5e4), (180 * u[2]).float()


def _images(xyz, frames, defocus, box, apix, g, trans=3, snr=0.05):
    """Normalised noisy particles: the atoms counted on the pixels of each frame's view, under the particle's CTF,
    moved by whole pixels, with white noise. [n, box, box] float32."""
    n = len(frames)
    out = torch.empty(n, box, box, device=DEV)
    for s in range(0, n, 256):
        f = frames[s:s + 256]
        k = len(f)
        xy = torch.round(torch.einsum("nij,aj->nai", f[:, :2], xyz) / apix).long() + box // 2
        ok = ((xy >= 0) & (xy < box)).all(-1)
        flat = (torch.arange(k, device=DEV)[:, None] * box + xy[..., 1]) * box + xy[..., 0]
        img = torch.bincount(flat[ok], minlength=k * box * box).reshape(k, box, box).double()
        spec = torch.fft.rfft2(img) * _ctf(box, apix, *(d[s:s + 256].double() for d in defocus))[1]
        img = torch.fft.irfft2(spec, s=(box, box)).float()
        shift = torch.randint(-trans, trans + 1, (k, 2), generator=g, device=DEV)
        row = (torch.arange(box, device=DEV)[None] - shift[:, :1]) % box
        col = (torch.arange(box, device=DEV)[None] - shift[:, 1:]) % box
        img = img[torch.arange(k, device=DEV)[:, None, None], row[:, :, None], col[:, None, :]]
        sd = img.std(dim=(1, 2), keepdim=True)
        img += torch.randn(img.shape, generator=g, device=DEV) * sd / math.sqrt(snr)
        out[s:s + 256] = (img - img.mean(dim=(1, 2), keepdim=True)) / img.std(dim=(1, 2), keepdim=True)
    return out


def _volume(n, g):
    """Blobs around the box centre and noise in every shell, [n]^3 float32."""
    ax = torch.arange(n, device=DEV, dtype=torch.float64)
    v = 0.2 * torch.randn(n, n, n, generator=g, device=DEV, dtype=torch.float64)
    u = torch.rand(6, 5, generator=g, device=DEV, dtype=torch.float64).cpu().numpy()
    for q in u:
        c, s = n / 2 + (q[:3] - 0.5) * n / 3, 1.5 + q[3] * (n / 16 - 1.5)
        e = [torch.exp(-(ax - ci) ** 2 / (2 * s * s)) for ci in c]
        v += (0.5 + 1.5 * q[4]) * e[0][:, None, None] * e[1][:, None] * e[2]
    return v.float()


def _model(case, seed):
    """Two chains and their PDB text, from the seed."""
    from gisapr_gb300 import synthetic as syn
    return syn.make_model(syn.residues_for_atoms(case["moving"]), syn.residues_for_atoms(case["fixed"]), int(seed))


def _poses(n, seed, rotation=3.0, translation=1.5):
    rng = np.random.default_rng(seed + 17)
    p = rng.normal(size=(n, 2, 3))
    p /= np.linalg.norm(p, axis=2, keepdims=True)
    p *= np.stack([rng.uniform(0, rotation, n), rng.uniform(0, translation, n)], 1)[..., None]
    return p.reshape(n, 6)


def _lists(rot, tilt, m_rot, m_tilt, reach):
    """Directions within ``reach`` degrees of each particle (rot, tilt and mean angle of the axes)."""
    e = _euler(m_rot, m_tilt, torch.zeros_like(m_rot))
    p = _euler(rot, tilt, torch.zeros_like(rot))
    near = (((m_rot[None] - rot[:, None] + 180) % 360 - 180).abs() <= reach) & ((m_tilt[None] - tilt[:, None]).abs() <= reach)
    near &= torch.rad2deg(torch.acos(torch.einsum("pik,dik->pdi", p, e).clamp(-1, 1))).mean(-1) <= reach
    near = near.cpu().numpy()
    return [np.nonzero(row)[0].tolist() for row in near]


def _search(case, seed):
    """Everything a search job is made from: model, particles (STAR angles near the true ones), directions, lists."""
    from gisapr_gb300 import synthetic as syn
    box = case["box"]
    apix, order, reach, step, crop, half_res = SEARCH[box]
    g = _gen(seed)
    model = _model(case, seed)
    n = case["particles"]
    rot, tilt = _directions(n, g)
    psi = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 360
    defocus = _defocus(n, g)
    xyz = torch.as_tensor(model.coords, device=DEV)
    images = _images(xyz, _euler(rot, tilt, psi), defocus, box, apix, g)
    off = torch.rand(3, n, generator=g, device=DEV, dtype=torch.float64) - 0.5
    rot, tilt = rot + reach * off[0], (tilt + reach * off[1]).clamp(0, 180)
    psi = (psi + step * off[2]) % 360
    m_rot, m_tilt = (np.asarray(v) for v in syn.healpix_directions(order))
    lists = _lists(rot, tilt, torch.as_tensor(m_rot, device=DEV), torch.as_tensor(m_tilt, device=DEV), reach)
    return dict(model=model, images=images, rot=rot.cpu().numpy(), tilt=tilt.cpu().numpy(), psi=psi.cpu().numpy(),
                defocus=defocus, m_rot=m_rot, m_tilt=m_tilt, lists=lists, apix=apix, reach=reach, step=step,
                crop=crop, fsc=_fsc(box, apix, half_res))


def _stack(case, seed):
    """A stack of particles, its in-plane angles and its CTF weights, for ``particles``."""
    g = _gen(seed)
    n, box, nb = case["n"], case["box"], case["newbox"]
    apix = SEARCH[box][0]
    rot, tilt = _directions(n, g)
    xyz = torch.randn(2000, 3, generator=g, device=DEV, dtype=torch.float64) * box * apix / 8
    psi = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 360
    defocus = _defocus(n, g)
    images = _images(xyz, _euler(rot, tilt, psi), defocus, box, apix, g)
    ctf = torch.empty(n, nb, nb // 2 + 1, device=DEV)
    for s in range(0, n, 256):
        ctf[s:s + 256] = _ctf(nb, apix * box / nb, *(d[s:s + 256].double() for d in defocus))[0].float()
    step = SEARCH[box][3]
    angles = [[_nudge(k * step) for k in range(i, i + case["psi"])] for i in (torch.round(psi / step).long() - case["psi"] // 2).tolist()]
    return images, ctf, angles


def _nudge(a):
    """The in-plane angle the search uses for a nominal one: half a degree in the place of zero."""
    return 0.5 if abs(a) < 0.5 else float(a)


def _spectra(case, seed):
    """Unit-norm templates of a smooth object and a noisy particle that holds one of them, for ``correlate``."""
    g = _gen(seed)
    n, h = case["box"], case["box"] // 2 + 1
    shape = (case["dirs"], n, h)
    common = torch.randn(1, n, h, 2, generator=g, device=DEV, dtype=torch.float64)
    t = torch.view_as_complex(common + torch.randn(*shape, 2, generator=g, device=DEV, dtype=torch.float64))
    t = t / t.abs().square().sum((-2, -1), keepdim=True).sqrt()
    p = torch.view_as_complex(torch.randn(case["psi"], n, h, 2, generator=g, device=DEV, dtype=torch.float64))
    p = p / p.abs().square().sum((-2, -1), keepdim=True).sqrt() + 0.05 * t[:1].conj()
    p = p / p.abs().square().sum((-2, -1), keepdim=True).sqrt()
    return t.to(torch.complex64), p.to(torch.complex64)


def _raw(case, seed):
    """Raw particles with a gradient, and their shifts, for ``ingest``."""
    g = _gen(seed)
    n, s = case["n"], case["size"]
    ramp = torch.linspace(-1, 1, s, device=DEV)
    img = torch.randn(n, s, s, generator=g, device=DEV) + 0.3 * ramp[:, None] + 0.2 * ramp + 4.0
    shifts = torch.rand(n, 2, generator=g, device=DEV, dtype=torch.float64) * 12 - 6
    return img, shifts.cpu().numpy()


# ---------------------------------------------------------------------------------------------- the calls


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("score", "generation"):
        from gisapr_gb300.engine import BatchScoringJob, JobConfig, ScoringJob
        from gisapr_gb300.tables import ParticleRecord, model_angles_from_lists
        d = _search(case, seed)
        du, dv, da = (v.tolist() for v in d["defocus"])
        records = [ParticleRecord(i + 20, "%d@stack.mrcs" % (i + 1), float(r), float(t), float(p), u, v, a)
                   for i, (r, t, p, u, v, a) in enumerate(zip(d["rot"], d["tilt"], d["psi"], du, dv, da))]
        cfg = JobConfig(box=case["box"], apix=d["apix"], crop=d["crop"], psi_step=d["step"], local_range=d["reach"])
        job = ScoringJob(cfg, d["model"].pdb_text, model_angles_from_lists(d["m_rot"].tolist(), d["m_tilt"].tolist()),
                         records, d["images"], fsc_values=d["fsc"], device=DEV, local=d["lists"])
        if kind == "score":
            return dict(kind=kind, job=job, pose=_poses(1, seed)[0])
        batch = BatchScoringJob(job, case["poses"], precision=case["precision"])
        return dict(kind=kind, job=job, batch=batch, poses=_poses(case["poses"], seed))
    if kind == "templates":
        from gisapr_gb300.search import IntegratedProjector, PackedFourierLayout
        from gisapr_gb300.tables import model_angles_from_lists
        g = _gen(seed)
        box, nb = case["box"], case["newbox"]
        rot, tilt = _directions(case["dirs"], g)
        mask = _soft_mask(box, round(0.43 * box)).float() if case["masked"] else None
        fsc = _packed_fsc(_fsc(box, SEARCH.get(box, (3.0,))[0], 4.0 if box > 32 else None), nb).float()
        projector = IntegratedProjector(DEV, box, nb, PackedFourierLayout(nb, 12, DEV), mask, fsc)
        return dict(kind=kind, projector=projector, volume=_volume(box, g),
                    angles=model_angles_from_lists(rot.tolist(), tilt.tolist()))
    if kind == "particles":
        from gisapr_gb300.search import PackedFourierLayout, ParticleFourierPreparer, PsiGridBank
        images, ctf, angles = _stack(case, seed)
        box, nb = case["box"], case["newbox"]
        bank = PsiGridBank(box, DEV, sorted({a for row in angles for a in row}))
        index = torch.tensor([[bank.angle_to_index[a] for a in row] for row in angles], dtype=torch.int32, device=DEV)
        mask = _soft_mask(box, round(0.43 * box)).float() if case["masked"] else None
        preparer = ParticleFourierPreparer(box, nb, DEV, PackedFourierLayout(nb, 12, DEV), mask, bank)
        return dict(kind=kind, preparer=preparer, images=images, index=index, ctf=ctf)
    if kind == "correlate":
        from gisapr_gb300.search import CorrelationWorkspace, PackedFourierLayout
        t, p = _spectra(case, seed)
        return dict(kind=kind, t=t, p=p, layout=PackedFourierLayout(case["box"], case["crop"], DEV),
                    work=CorrelationWorkspace(DEV))
    if kind == "density":
        from gisapr_gb300.pdb2mrc import MovedChainDensity
        model = MovedChainDensity(_model(case, seed).pdb_text, "A", case["box"], case["apix"], 2 * case["apix"], DEV,
                                  from_text=True)
        return dict(kind=kind, model=model, pose=_poses(1, seed)[0])
    if kind == "ingest":
        images, shifts = _raw(case, seed)
        return dict(kind=kind, images=images, shifts=shifts, case=dict(case))
    from gisapr_gb300.restraint import GeometryRestraint
    fd, path = tempfile.mkstemp(suffix=".pdb")
    with os.fdopen(fd, "w") as f:
        f.write(_body(case, seed)[0])
    restraint = GeometryRestraint(path, "A", DEV, boxsize=case["box"], apix=case["apix"])
    os.unlink(path)
    return dict(kind="restraint", restraint=restraint, poses=_poses(case["poses"], seed, 20.0, 6.0))


def _body(case, seed):
    """PDB text with chain A moved out of the main body, half of the poses' reach away from touching it."""
    model = _model(case, seed)
    moved = model.coords[model.moving]
    reach = np.abs(model.coords[~model.moving]).max() * 0.8
    out, k = [], 0
    for line in model.pdb_text.splitlines(keepends=True):
        if line[21:22] == "A" and line.startswith("ATOM"):
            x, y, z = moved[k] + (reach, 0.0, 0.0)
            line = "%s%8.3f%8.3f%8.3f%s" % (line[:30], x, y, z, line[54:])
            k += 1
        out.append(line)
    return "".join(out), model, reach


def run(state):
    kind = state["kind"]
    if kind == "score":
        job = state["job"]
        score = job.score(state["pose"])
        return dict(score=score, peak=job.peak, zscore=job.zscore)
    if kind == "generation":
        batch = state["batch"]
        scores = batch.score_batch(state["poses"])
        return dict(scores=scores.astype(np.float32), peak=batch.peak, zscore=batch.zscore)
    if kind == "templates":
        return state["projector"].build_templates(state["volume"], state["angles"])
    if kind == "particles":
        return state["preparer"].prepare_batch(state["images"], state["index"], state["ctf"])
    if kind == "correlate":
        from gisapr_gb300.search import correlate_templates_and_particle
        return correlate_templates_and_particle(state["t"], state["p"], state["layout"], state["work"])
    if kind == "density":
        return state["model"].generate(state["pose"])
    if kind == "ingest":
        from gisapr_gb300.ingest import preprocess_stack
        c = state["case"]
        return preprocess_stack(state["images"], state["shifts"], c["crop"], c["whitening"], c["highpass"], 50.0, 1.1)
    return state["restraint"].evaluate_many(state["poses"])


# ------------------------------------------------------------------------------------------ least work of a pass


def _fft2(n):
    """Operations of one real n x n transform."""
    return 2.5 * n * n * 2 * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind in ("score", "generation"):
        n, k = case["box"], case["box"] * (case["box"] // 2 + 1)
        _, order, reach, step, crop, _ = SEARCH[n]
        psi = 2 * int(reach // step) + 1
        dirs = 12 * 4 ** order
        maps = case["particles"] * psi * (5.6 if n >= 96 else 3.1)  # mean length of the local lists
        splat = (case["moving"]) * 12.0 ** 3 * 20
        per_map = 6 * k + 5 * (n // 2 + 1) * n * 2 + 4 * crop * crop * (n // 2 + 1)
        spectrum = 2.5 * (2 * n) ** 3 * 3 * math.log2(2 * n)
        one = splat + spectrum + dirs * (8 * n * n * 10 + 4 * _fft2(n)) + maps * per_map
        c = case.get("poses", 1)
        stack = case["particles"] * psi * k * 8
        return dict(bytes=stack + c * (case["particles"] * 12.0 + case["moving"] * 16) + 4 * n ** 3, flops=c * one)
    if kind == "templates":
        n, nb, d = case["box"], case["newbox"], case["dirs"]
        spectrum = 2.5 * (2 * n) ** 3 * 3 * math.log2(2 * n)
        return dict(bytes=4.0 * n ** 3 + 8.0 * d * nb * (nb // 2 + 1),
                    flops=spectrum + d * (2 * n * n * 30 + _fft2(2 * n) / 2 + 3 * _fft2(n)))
    if kind == "particles":
        n, nb, m = case["box"], case["newbox"], case["n"] * case["psi"]
        h = nb // 2 + 1
        return dict(bytes=4.0 * case["n"] * (n * n + nb * h) + 8.0 * m * nb * h, flops=m * (_fft2(n) + 20.0 * n * n))
    if kind == "correlate":
        n, h, c, maps = case["box"], case["box"] // 2 + 1, case["crop"], case["dirs"] * case["psi"]
        return dict(bytes=8.0 * (case["dirs"] + case["psi"]) * n * h + 20.0 * maps,
                    flops=maps * (6.0 * n * h + 10.0 * n * h + 4.0 * c * c * h))
    if kind == "density":
        return dict(bytes=8.0 * case["box"] ** 3 + 16.0 * case["moving"], flops=case["moving"] * 12.0 ** 3 * 20)
    if kind == "ingest":
        c = case["crop"] or case["size"]
        steps = 1 + (2 if case["whitening"] else 0) + (2 if case["highpass"] else 0)
        return dict(bytes=8.0 * case["n"] * c * c, flops=case["n"] * (steps * _fft2(c) + 20.0 * c * c))
    # the voxels of the moved chain: about 8 A^3 an atom, and the density of its atoms
    voxels = case["moving"] * 20.0 / case["apix"] ** 3
    return dict(bytes=case["poses"] * (voxels * 5 + case["moving"] * 16.0), flops=case["poses"] * case["moving"] * 12.0 ** 3 * 20)


# ------------------------------------------------------------------------------------- the same results in 64 bits

_Z = {"H": 1.0, "C": 6.0, "N": 7.0, "O": 8.0, "P": 15.0, "S": 16.0}


def _x_rotation(pose):
    """Matrix of the pose's rotation vector (degrees), by Rodrigues' formula."""
    v = np.deg2rad(np.asarray(pose[:3], dtype=np.float64))
    a = np.linalg.norm(v)
    if a == 0:
        return np.eye(3)
    x, y, z = v / a
    k = np.array([[0, -z, y], [z, 0, -x], [-y, x, 0]])
    return np.eye(3) + math.sin(a) * k + (1 - math.cos(a)) * (k @ k)


def _x_density(xyz, z, box, apix):
    """sum of Z kn exp(-rp r) over each atom's cube, [z, y, x] float64."""
    res = 2 * apix
    w = int(round(res * 3 / apix))
    rp = (math.pi * apix / res) ** 2
    kn = (rp / math.pi) ** 1.5
    pos = torch.as_tensor(xyz, device=DEV, dtype=torch.float64) / apix + box // 2
    pos = pos.float().double()
    lo = torch.floor((pos - w).abs() + 0.5) * torch.sign(pos - w)
    hi = torch.floor((pos + w).abs() + 0.5) * torch.sign(pos + w)
    lo, hi = lo.clamp(min=0).long(), hi.clamp(max=box - 1).long()
    ax = torch.arange(2 * w + 2, device=DEV)
    out = torch.zeros(box ** 3, device=DEV, dtype=torch.float64)
    zk = torch.as_tensor(z, device=DEV, dtype=torch.float64) * kn
    for s in range(0, len(pos), 2000):
        v = [lo[s:s + 2000, i, None] + ax for i in range(3)]
        ok = [v[i] < hi[s:s + 2000, i, None] for i in range(3)]
        d = [(v[i] - pos[s:s + 2000, i, None]) ** 2 for i in range(3)]
        r = (d[2][:, :, None, None] + d[1][:, None, :, None] + d[0][:, None, None, :]).sqrt()
        m = ok[2][:, :, None, None] & ok[1][:, None, :, None] & ok[0][:, None, None, :]
        idx = (v[2][:, :, None, None] * box + v[1][:, None, :, None]) * box + v[0][:, None, None, :]
        val = zk[s:s + 2000, None, None, None] * torch.exp(-rp * r)
        out.index_add_(0, idx[m], val[m])
    return out.reshape(box, box, box)


def _x_moved(model, pose):
    """Coordinates of all atoms with chain A moved, its coordinates written and read back with three decimals."""
    sel = model.moving
    xyz = model.coords.astype(np.float32)
    pivot = np.mean(xyz[sel], axis=0).astype(np.float64)
    m = (xyz[sel].astype(np.float64) - pivot) @ _x_rotation(pose) + pivot + pose[3:]
    out = xyz.astype(np.float64)
    out[sel] = np.rint(m * 1000) / 1000
    return out.astype(np.float32), np.array([_Z[e] for e in model.elements])


def _x_templates(volume, rot, tilt, nb, mask, fsc):
    """Templates of one density, [dirs, nb, nb/2+1] complex128, stored shifted."""
    n = volume.shape[0]
    m = 2 * n
    f = torch.fft.fftshift(torch.fft.fftfreq(m, device=DEV, dtype=torch.float64))
    vol = torch.nn.functional.pad(volume.double(), [n // 2] * 6)
    q = f * f
    vol *= torch.sinc((q[:, None, None] + q[:, None] + q).sqrt()) ** 2
    dft = torch.fft.fftshift(torch.fft.rfftn(torch.fft.fftshift(vol)), dim=(0, 1)).contiguous()
    del vol
    R = _euler(rot, tilt, torch.zeros_like(rot)).float().double()  # the angle table keeps float32 matrices
    gx = torch.arange(n + 1, device=DEV, dtype=torch.float64)[None, :]
    gy = torch.fft.ifftshift(f)[:, None] * m
    i = torch.arange(n, device=DEV)
    shell = torch.round(torch.sqrt(((i - n // 2)[:, None] ** 2 + (i - n // 2) ** 2).double())).long()
    shell = torch.fft.ifftshift(shell)
    count = torch.bincount(shell.reshape(-1)).double()
    k = torch.arange(n, device=DEV, dtype=torch.float64) - (n - 1) / 2
    kk = (k * k).sum() * n
    h = nb // 2 + 1
    out = torch.empty(len(R), nb, h, device=DEV, dtype=torch.complex128)
    step = max(1, 2 ** 22 // (m * (n + 1)))
    rows = torch.cat((torch.arange(nb // 2, device=DEV), torch.arange(n - nb // 2, n, device=DEV)))
    for s in range(0, len(R), step):
        r = R[s:s + step].transpose(1, 2)  # columns of the frame: (x, y, z) = (row 0, row 1) combined
        x, y, z = (r[:, a, 0, None, None] * gx + r[:, a, 1, None, None] * gy for a in range(3))
        neg = x < 0
        sign = torch.where(neg, -1.0, 1.0)
        cz, cy = ((c * sign + n).clamp(0, m - 1) for c in (z, y))
        cx = (x * sign).clamp(0, n)
        z0, y0, x0 = (c.floor().long() for c in (cz, cy, cx))
        val = 0
        for dz in (0, 1):
            for dy in (0, 1):
                for dx in (0, 1):
                    wt = ((cz - z0 if dz else 1 - cz + z0) * (cy - y0 if dy else 1 - cy + y0)
                          * (cx - x0 if dx else 1 - cx + x0))
                    at = ((z0 + dz).clamp(max=m - 1) * m + (y0 + dy).clamp(max=m - 1)) * (n + 1) + (x0 + dx).clamp(max=n)
                    val = val + wt * dft.reshape(-1)[at]
        val = torch.where(neg, val.conj(), val)
        img = torch.fft.ifftshift(torch.fft.irfft2(val, s=(m, m)), dim=(1, 2))[:, n // 2:n // 2 + n, n // 2:n // 2 + n]
        spec = torch.fft.fft2(img)
        amp = torch.zeros(len(spec), len(count), device=DEV, dtype=torch.float64)
        amp.index_add_(1, shell.reshape(-1), spec.abs().reshape(len(spec), -1))
        div = count / amp
        div[:, 0] = 1
        img = torch.fft.ifft2(spec * div[:, shell]).real
        a = (img * k[:, None]).sum((1, 2)) / kk
        b = (img * k).sum((1, 2)) / kk
        img = img - img.mean((1, 2), keepdim=True) - a[:, None, None] * k[:, None] - b[:, None, None] * k
        img = img / img.square().mean((1, 2), keepdim=True).sqrt()
        if mask is not None:
            img = img * mask
        out[s:s + step] = _x_pack(torch.fft.fft2(img), rows, nb) * fsc
    out /= out.abs().square().sum((1, 2), keepdim=True).sqrt()
    return torch.fft.fftshift(out, dim=(1, 2))


def _x_pack(full, rows, nb):
    """The packed nb x (nb/2+1) half plane of full transforms (its last column is the negative Nyquist one)."""
    n = full.shape[-1]
    cols = torch.cat((torch.arange(nb // 2, device=DEV), torch.tensor([n - nb // 2], device=DEV)))
    return full[:, rows][:, :, cols]


def _x_particles(images, angles, ctf, nb, mask):
    """Rotated, masked, weighted, conjugated and normalised spectra, [n, psi, nb, nb/2+1] complex128, shifted."""
    n, box = images.shape[0], images.shape[-1]
    ax = torch.arange(box, device=DEV, dtype=torch.float64) - box / 2
    th = torch.deg2rad(torch.tensor(angles, device=DEV, dtype=torch.float64))
    out = torch.empty(*th.shape, nb, nb // 2 + 1, device=DEV, dtype=torch.complex128)
    rows = torch.cat((torch.arange(nb // 2, device=DEV), torch.arange(box - nb // 2, box, device=DEV)))
    step = max(1, 2 ** 22 // (box * box))
    for s in range(0, n, step):
        img = images[s:s + step].double()
        img = torch.nn.functional.pad(img, [1, 2, 1, 2])
        flat = img.reshape(len(img), -1)
        for q in range(th.shape[1]):
            c, sn = th[s:s + step, q].cos()[:, None, None], th[s:s + step, q].sin()[:, None, None]
            sy = (c * ax[:, None] - sn * ax + box / 2).clamp(-1, box)
            sx = (sn * ax[:, None] + c * ax + box / 2).clamp(-1, box)
            y0, x0 = sy.floor(), sx.floor()
            ty, tx = sy - y0, sx - x0
            at = ((y0.long() + 1) * (box + 3) + x0.long() + 1).reshape(len(img), -1)
            v = 0
            for dy, wy in ((0, 1 - ty), (1, ty)):
                for dx, wx in ((0, 1 - tx), (1, tx)):
                    v = v + wy * wx * flat.gather(1, at + dy * (box + 3) + dx).reshape(-1, box, box)
            if mask is not None:
                v = v * mask
            p = (_x_pack(torch.fft.fft2(v), rows, nb) * ctf[s:s + step].double()).conj()
            out[s:s + step, q] = p / p.abs().square().sum((1, 2), keepdim=True).sqrt()
    return torch.fft.fftshift(out, dim=(2, 3))


def _x_twiddles(n, crop):
    off = torch.arange(crop, device=DEV, dtype=torch.float64) - crop // 2
    r = torch.arange(n, device=DEV, dtype=torch.float64)
    w = torch.full((n // 2 + 1,), 2.0, device=DEV, dtype=torch.float64)
    w[0] = w[n // 2] = 1
    ey = torch.exp(2j * math.pi * r[:, None] * off / n)
    return ey, w[:, None] * torch.exp(2j * math.pi * r[: n // 2 + 1, None] * off / n)


def _x_maps(t, p, ey, ex):
    """Correlation windows of templates [b, d, r, c] and spectra [b, s, r, c]: [b, d, s, y, x] float64."""
    b, d, r, c = t.shape
    s, y = p.shape[1], ey.shape[1]
    u = (p.permute(0, 3, 2, 1)[..., None] * ey[:, None, :]).reshape(b, c, r, s * y)
    zz = (t.permute(0, 3, 1, 2) @ u).reshape(b, c, d, s, y)
    return torch.einsum("bcdsy,cx->bdsyx", zz, ex).real


def _x_search(case, seed):
    d = _search(case, seed)
    box, n = case["box"], case["particles"]
    poses = _poses(case.get("poses", 1), seed)
    psi = np.array([[(round(((a + 360) % 360) / d["step"]) * d["step"]) % 360 + k * d["step"]
                     for k in range(-int(d["reach"] // d["step"]), int(d["reach"] // d["step"]) + 1)] for a in d["psi"]])
    angles = [[_nudge(a) for a in row] for row in psi]
    mask = _soft_mask(box, round(0.43 * box))
    fsc = _packed_fsc(d["fsc"], box)
    rot, tilt = (torch.as_tensor(v, device=DEV) for v in (d["m_rot"], d["m_tilt"]))
    ey, ex = _x_twiddles(box, d["crop"])
    spectra = torch.cat([_x_particles(d["images"][s:s + 500], angles[s:s + 500],
                                      _ctf(box, d["apix"], *(v[s:s + 500].double() for v in d["defocus"]))[0], box, mask)
                         for s in range(0, n, 500)])
    count = torch.tensor([len(v) for v in d["lists"]], device=DEV)
    most = max(1, int(count.max()))
    lists = torch.tensor([v + [0] * (most - len(v)) for v in d["lists"]], device=DEV)
    listed = torch.arange(most, device=DEV) < count[:, None]
    peak = torch.zeros(len(poses), n, device=DEV, dtype=torch.float64)
    z = torch.zeros_like(peak)
    for c, pose in enumerate(poses):
        bank = _x_templates(_x_density(*_x_moved(d["model"], pose), box, d["apix"]), rot, tilt, box, mask, fsc)
        for s in range(0, n, 40):
            top = _x_maps(bank[lists[s:s + 40]], spectra[s:s + 40], ey, ex).amax((-2, -1)) * 1024
            ok = listed[s:s + 40, :, None].expand_as(top)
            k = ok.sum((1, 2)).clamp(min=1)
            mean = torch.where(ok, top, 0.0).sum((1, 2)) / k
            sd = (torch.where(ok, (top - mean[:, None, None]) ** 2, 0.0).sum((1, 2)) / k).sqrt()
            best = torch.where(ok, top, -math.inf).amax((1, 2))
            some = count[s:s + 40] > 0
            peak[c, s:s + 40] = torch.where(some, best, 0.0)
            z[c, s:s + 40] = torch.where(some, (best - mean) / sd, 0.0)
    scores = torch.where(count > 0, torch.exp(peak / 1024), 0.0).sum(1)
    if case["kind"] == "score":
        return dict(score=float(scores[0]), peak=peak[0], zscore=z[0])
    return dict(scores=scores, peak=peak, zscore=z)


def _x_distance(mask):
    """Squared distance of every voxel to the nearest set one, one axis after another (float64, exact integers)."""
    n = mask.shape[0]
    i = torch.arange(n, device=DEV, dtype=torch.float32)
    sq = (i[:, None] - i) ** 2
    f = torch.where(mask, 0.0, 1e9).float()
    for axis in (2, 1, 0):
        rows = f.movedim(axis, 2).reshape(-1, n)
        rows = torch.cat([(rows[s:s + 2048, None, :] + sq).amin(2) for s in range(0, len(rows), 2048)])
        f = rows.reshape(n, n, n).movedim(2, axis)
    return f.double()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("score", "generation"):
        if case.get("poses", 1) * (case["particles"] * (case["box"] / 128) ** 2 + 300) > 30000:
            return None  # over about 20 seconds
        return _x_search(case, seed)
    if kind == "templates":
        g = _gen(seed)
        box, nb = case["box"], case["newbox"]
        rot, tilt = _directions(case["dirs"], g)
        mask = _soft_mask(box, round(0.43 * box)).float().double() if case["masked"] else None
        fsc = _packed_fsc(_fsc(box, SEARCH.get(box, (3.0,))[0], 4.0 if box > 32 else None), nb)
        return _x_templates(_volume(box, g), rot, tilt, nb, mask, fsc)
    if kind == "particles":
        images, ctf, angles = _stack(case, seed)
        mask = _soft_mask(case["box"], round(0.43 * case["box"])).float().double() if case["masked"] else None
        return _x_particles(images, angles, ctf, case["newbox"], mask)
    if kind == "correlate":
        t, p = _spectra(case, seed)
        raw = _x_maps(t[None].to(torch.complex128), p[None].to(torch.complex128), *_x_twiddles(case["box"], case["crop"]))[0]
        best, at = raw.reshape(*raw.shape[:2], -1).max(-1)
        return best * 1024, at // case["crop"], at % case["crop"]
    if kind == "density":
        model = _model(case, seed)
        return _x_density(*_x_moved(model, _poses(1, seed)[0]), case["box"], case["apix"])
    if kind == "ingest":
        img, shifts = _raw(case, seed)
        n, s, c = case["n"], case["size"], case["crop"] or case["size"]
        sh = torch.as_tensor(np.floor(shifts + 0.5), device=DEV).long()
        at = torch.arange(c, device=DEV) + s // 2 - c // 2
        col, row = (at[None] - sh[:, a, None] for a in (0, 1))
        ok = ((row >= 0) & (row < s))[:, :, None] & ((col >= 0) & (col < s))[:, None]
        v = img[torch.arange(n, device=DEV)[:, None, None], row.clamp(0, s - 1)[:, :, None], col.clamp(0, s - 1)[:, None]]
        v = torch.where(ok, v, 0.0).double()
        i = torch.arange(c, device=DEV) - c // 2
        r = (i[:, None] ** 2 + i[None] ** 2).double().sqrt()
        if case["whitening"]:
            shell = torch.fft.ifftshift(torch.round(r).long())
            count = torch.bincount(shell.reshape(-1)).double()
            spec = torch.fft.fft2(v)
            amp = torch.zeros(n, len(count), device=DEV, dtype=torch.float64)
            amp.index_add_(1, shell.reshape(-1), spec.abs().reshape(n, -1))
            div = count / amp
            div[:, 0] = 1
            v = torch.fft.ifft2(spec * div[:, shell]).real
            k = torch.arange(c, device=DEV, dtype=torch.float64) - (c - 1) / 2
            kk = (k * k).sum() * c
            v = v - v.mean((1, 2), keepdim=True) - k[:, None] * (v * k[:, None]).sum((1, 2), keepdim=True) / kk \
                - k * (v * k).sum((1, 2), keepdim=True) / kk
            v = v / v.square().mean((1, 2), keepdim=True).sqrt()
        if case["highpass"]:
            f = r / c
            ring = round(c * 1.1 / 50.0)
            lo, hi = max(0.0, (ring - 2) / c), min(c, (ring + 2) / c)
            m = torch.where(f < lo, 0.0, torch.where(f <= hi, 0.5 - 0.5 * torch.cos(math.pi * (f - lo) / (hi - lo)), 1.0))
            v = torch.fft.ifft2(torch.fft.fft2(v) * torch.fft.ifftshift(m)).real
        return v
    _, model, reach = _body(case, seed)
    sel, box, apix = model.moving, case["box"], case["apix"]
    z = np.array([_Z[e] for e in model.elements])
    body = _x_density(model.coords[~sel].astype(np.float32), z[~sel], box, apix) > 1.0
    d2 = _x_distance(body)
    chain = np.round(model.coords[sel] + (reach, 0.0, 0.0), 3).astype(np.float32).astype(np.float64)
    centre = chain.mean(0)
    out = []
    for p in _poses(case["poses"], seed, 20.0, 6.0):
        q = (chain - centre) @ _x_rotation(p) + centre + p[3:]
        on = _x_density(q.astype(np.float32), z[sel], box, apix) > 1.0
        hits = int((on & body).sum())
        out.append((hits, float(d2[on].min().sqrt()) * apix if bool(on.any()) else None))
    return out
