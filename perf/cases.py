"""The work a user of the library has it do, as cases that can be timed and checked.

A case is a dict of plain values; its "kind" names the entry point it goes
through and the other values are sizes.  `prepare` makes what a program holds
before the call (atoms, transmission functions, waves, the context it keeps for
its whole run), `run` is one pass through a public entry point, `work` the
bytes and operations that pass cannot do without, and `exact` the same result
in 64 bits by plain torch.

Sizes are those of the five workloads (Si CTEM at 256^2, the SrTiO3 STEM scan
at 512^2, the uneven batch of jobs with sides 256 to 1024, Au frozen phonons at
2048^2, the learned coarse-slice closure at 256^2 and 512^2) and, for `draw`,
of the ranges around them that the library accepts.
"""
import math
import os

import numpy as np
import torch

from multislice_gb300 import Context
from multislice_gb300 import specimen as S
from multislice_gb300.api import Closure

DATA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multislice_gb300", "data")
SIDES = (64, 128, 256, 384, 512, 768, 1024, 2048)
DEV = "cuda"
CS, DF = 1.2e7, -600.0  # objective lens of the Au workload: 1.2 mm, -60 nm (Angstrom)


def listed():
    return [
        # one exit wave's spectrum: the smallest call a program makes, all latency
        dict(name="fft_256", kind="fft", nx=256, ny=256, batch=1),
        # the CTEM workload: Si, 80 slices, one plane wave, exit wave to the host
        dict(name="ctem_si_256", kind="ctem", nx=256, ny=256, nslice=80),
        # a partially coherent CTEM image: every illumination angle, defocus spread
        dict(name="partial_256", kind="partial", nx=256, ny=256, nslice=20, mrad=2.0, spread=60.0),
        # the STEM workload's stages: projected potentials of 100 slices ...
        dict(name="potential_srtio3_512", kind="potential", crystal="srtio3", cells=8, nslice=100, nx=512, ny=512,
             radius=5.0),
        # ... and the scan itself, a quarter of the raster through a fifth of the crystal
        dict(name="stem_512", kind="stem", nx=512, ny=512, nprobe=1024, nslice=20, ndet=2, ncheck=1),
        # entrance-to-exit waves of a scan on a mixed-radix, ragged grid
        dict(name="exit_waves_384", kind="exit", nx=384, ny=384, nprobe=61, nslice=12),
        # the uneven batch: sides 256 to 1024, plane waves and probes mixed
        dict(name="jobs_uneven", kind="jobs", njobs=20, max_slices=48),
        # transmission functions of a thick 1024^2 specimen
        dict(name="transmission_1024", kind="transmission", nx=1024, ny=1024, nlayer=24),
        # the frozen-phonon workload's stages: potentials of one Au configuration ...
        dict(name="potential_au_2048", kind="potential", crystal="au", cells=16, nslice=40, nx=2048, ny=2048,
             radius=3.0),
        # ... and several configurations' waves through the slice loop
        dict(name="waves_2048", kind="waves", nx=2048, ny=2048, batch=8, nslice=6),
        # the closure on the exit waves of a 512^2 scan, and one training gradient at 256^2
        dict(name="closure_apply_512", kind="apply", batch=16, h=512, w=512),
        dict(name="closure_grad_256", kind="grad", batch=8, h=256, w=256),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    """One more case of the listed ones' ranges: any entry point, sizes spread over what it takes."""
    kind = rng.choice(["fft", "ctem", "partial", "potential", "stem", "exit", "jobs", "transmission", "waves", "apply",
                       "grad"])
    if kind == "fft":
        nx, ny = rng.choice(SIDES), rng.choice(SIDES)
        return dict(kind=kind, nx=nx, ny=ny, batch=_log(rng, 1, max(1, min(200, (1 << 25) // (nx * ny)))))
    if kind == "ctem":
        n = rng.choice((64, 128, 256, 384, 512, 768))
        return dict(kind=kind, nx=n, ny=rng.choice((n, n, n, 128, 256)), nslice=_log(rng, 3, 120))
    if kind == "partial":
        return dict(kind=kind, nx=rng.choice((128, 256)), ny=rng.choice((128, 256)), nslice=_log(rng, 3, 20),
                    mrad=rng.uniform(0.5, 2.0), spread=rng.choice((0.0, 30.0, 60.0)))
    if kind == "potential":
        crystal = rng.choice(("si", "srtio3", "au"))
        nx, ny = rng.choice(SIDES[1:]), rng.choice(SIDES[1:])
        return dict(kind=kind, crystal=crystal, cells=rng.randint(4, 12), nx=nx, ny=ny, radius=rng.uniform(2.5, 5.0),
                    nslice=_log(rng, 1, max(1, min(100, (1 << 26) // (nx * ny)))))
    if kind == "stem":
        n = rng.choice((256, 512))
        return dict(kind=kind, nx=n, ny=rng.choice((n, 256, 512)), nprobe=_log(rng, 1, 900), nslice=_log(rng, 2, 20),
                    ndet=rng.randint(1, 4), ncheck=rng.randint(1, 2))
    if kind == "exit":
        nx, ny = rng.choice(SIDES[1:]), rng.choice(SIDES[1:])
        return dict(kind=kind, nx=nx, ny=ny, nprobe=_log(rng, 1, max(1, min(300, (1 << 24) // (nx * ny)))),
                    nslice=_log(rng, 2, 16))
    if kind == "jobs":
        return dict(kind=kind, njobs=_log(rng, 2, 18), max_slices=rng.randint(22, 44))
    if kind == "transmission":
        nx, ny = rng.choice(SIDES), rng.choice(SIDES)
        return dict(kind=kind, nx=nx, ny=ny, nlayer=_log(rng, 1, max(1, min(100, (1 << 24) // (nx * ny)))))
    if kind == "waves":
        nx, ny = rng.choice(SIDES[2:]), rng.choice(SIDES[2:])
        return dict(kind=kind, nx=nx, ny=ny, batch=_log(rng, 1, max(1, min(64, (1 << 24) // (nx * ny)))),
                    nslice=rng.randint(2, 6))
    b = _log(rng, 1, 14)
    return dict(kind=kind, batch=b if kind == "apply" else min(b, 8), h=rng.randint(64, 512 if kind == "apply" else 256),
                w=128 * rng.randint(1, 4 if kind == "apply" else 2))


# ------------------------------------------------------------------- inputs
_ctx = None


def context():
    """The one context a program keeps for all its calls."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def layers(nx, ny, ax, by, kev, n, seed):
    """Band-limited transmission functions exp(i sigma V) of n layers of atoms at
    random sites (one per 4 A^2, peaks of some hundred V*A), complex64 [n, nx, ny]."""
    g = _gen(seed)
    kx = torch.fft.fftfreq(nx, ax / nx, device=DEV, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, by / ny, device=DEV, dtype=torch.float64)
    k2 = kx[:, None] ** 2 + ky[None, :] ** 2
    form = 1.0 / (1.0 + k2 / 0.25) ** 2  # peaked and screened, as an atom's scattering factor
    kmax = min(nx / (2 * ax), ny / (2 * by)) * 2 / 3
    natom = max(4, int(ax * by / 4.0))
    t = torch.empty((n, nx, ny), dtype=torch.complex64, device=DEV)
    for i in range(n):
        v = torch.zeros(nx * ny, dtype=torch.float64, device=DEV)
        site = torch.randint(0, nx * ny, (natom,), generator=g, device=DEV)
        v.index_add_(0, site, torch.ones(natom, dtype=torch.float64, device=DEV))
        v = torch.fft.ifft2(torch.fft.fft2(v.view(nx, ny)) * form).real * (40.0 * 14.0 * nx * ny / (ax * by))
        t[i] = torch.fft.ifft2(torch.fft.fft2(torch.exp(1j * sigma_kv(kev) * 1e-3 * v)) * (k2 < kmax * kmax))
    return t


def crystal(case, seed):
    """A crystal with thermal displacements of 0.08 A, as thick as its slices ask for."""
    n = case["cells"]
    make, per = {"si": (S.si_diamond, 4), "srtio3": (S.srtio3, 2), "au": (S.fcc_au, 2)}[case["crystal"]]
    spec = make(n, n, -(-case["nslice"] // per))
    spec = S.jitter(spec, 0.08, np.random.default_rng(seed))
    spec.cz = spec.cz * case["nslice"] / (per * -(-case["nslice"] // per))
    return spec


def _complex(shape, seed):
    return torch.randn(shape, dtype=torch.complex64, device=DEV, generator=_gen(seed))


def probe_like(batch, h, w, seed):
    """Waves like a scan's exit waves: a spot a few pixels wide on a weak, structured background."""
    z = _complex((batch, h, w), seed)
    kx = torch.fft.fftfreq(h, device=DEV)[:, None]
    ky = torch.fft.fftfreq(w, device=DEV)[None, :]
    z = torch.fft.ifft2(torch.fft.fft2(z) * torch.exp(-(kx ** 2 + ky ** 2) / (2 * 0.08 ** 2)))
    y = (torch.arange(h, device=DEV) - h / 2)[:, None]
    x = (torch.arange(w, device=DEV) - w / 2)[None, :]
    return (z * (0.05 + torch.exp(-(x * x + y * y) / (2 * 20.0 ** 2)))).to(torch.complex64)


def cell(case):
    """Cell edges: 0.06 A pixels (the STEM and closure workloads) or 0.106 A (the CTEM
    workload) along x, a little more along y."""
    px = 0.106 if case["kind"] in ("ctem", "partial") else 0.061
    return px * case["nx"], px * case["ny"] * 1.03


def _scan(case, seed):
    ax, by = cell(case)
    rng = np.random.default_rng(seed + 3)
    xy = rng.uniform(0.2, 0.8, (case["nprobe"], 2)) * (ax, by)
    return dict(k_ap=float(S.mrad_to_k(25.0, 200.0)), xy=xy)


DETECTORS = ((80.0, 200.0), (11.0, 22.0), (0.0, 11.0), (30.0, 70.0))  # mrad: HAADF, ABF, BF, LAADF


def job_list(case, seed):
    rng = np.random.default_rng(seed)
    jobs = []
    for j in range(case["njobs"]):
        n = (256, 384, 512, 768, 1024)[j % 5]
        ns = int(rng.integers(20, case["max_slices"] + 1))
        kev = float(rng.choice([80.0, 200.0, 300.0]))
        box = 0.1 * n
        nt = min(ns, 8)
        d = dict(trans=layers(n, n, box, box, kev, nt, seed * 1000 + j), ax=box, by=box, kev=kev,
                 dz=float(rng.uniform(1.0, 2.0)), layer_seq=rng.integers(0, nt, ns),
                 out=torch.empty((n, n), dtype=torch.complex64, device=DEV))
        if rng.random() < 0.5:
            d["probe"] = (float(S.mrad_to_k(rng.uniform(10.0, 30.0), kev)), float(rng.uniform(0, box)),
                          float(rng.uniform(0, box)))
        jobs.append(d)
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, ctx=context())
    if kind == "fft":
        st["psi"] = _complex((case["batch"], case["nx"], case["ny"]), seed)
        st["dir"] = 1
    elif kind in ("ctem", "partial", "stem", "exit", "waves"):
        ax, by = cell(case)
        nt = min(case["nslice"], 16)
        st["t"] = layers(case["nx"], case["ny"], ax, by, 200.0, nt, seed)
        rng = np.random.default_rng(seed + 1)
        st["seq"] = rng.integers(0, nt, case["nslice"])
        st["dz"] = rng.uniform(1.2, 2.0, nt)
        if kind in ("stem", "exit"):
            st.update(_scan(case, seed))
        if kind == "stem":
            st["det"] = [tuple(float(S.mrad_to_k(m, 200.0)) for m in d) for d in DETECTORS[:case["ndet"]]]
            last = case["nslice"] - 1
            st["cps"] = [last] if case["ncheck"] == 1 else [last // 2, last]
        if kind == "exit":
            st["out"] = torch.empty((case["nprobe"], case["nx"], case["ny"]), dtype=torch.complex64, device=DEV)
        if kind == "waves":
            st["psi"] = torch.exp(1j * 0.1 * _complex((case["batch"], case["nx"], case["ny"]), seed + 2).real)
    elif kind == "potential":
        st["spec"] = crystal(case, seed)
        st["out"] = torch.empty((case["nslice"], case["nx"], case["ny"]), dtype=torch.float32, device=DEV)
    elif kind == "transmission":
        shape = (case["nlayer"], case["nx"], case["ny"])
        v = torch.rand(shape, generator=_gen(seed), device=DEV)
        st["v"] = 2500.0 * v ** 30 + 20.0 * v  # a low background and few high peaks, as atoms make
        st["out"] = torch.empty(shape, dtype=torch.complex64, device=DEV)
    elif kind == "jobs":
        st["jobs"] = job_list(case, seed)
    else:
        st["net"] = Closure(st["ctx"], seed=1)
        st["net"].set_params(np.load(os.path.join(DATA, "closure_srtio3.npy")))
        st["psi"] = probe_like(case["batch"], case["h"], case["w"], seed)
        if kind == "grad":
            z = probe_like(case["batch"], case["h"], case["w"], seed + 1)
            st["fine"] = st["psi"] + 0.1 * z
    return st


# --------------------------------------------------------------------- pass
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "fft":
        # to reciprocal space and back, in turn, as a program between two filters
        psi = ctx.fft2d(st["psi"], 10.0, 10.0, st["dir"])
        st["dir"] = -st["dir"]
        return psi
    if kind == "potential":
        return ctx.potential(st["spec"], case["nx"], case["ny"], case["nslice"], case["radius"], out=st["out"])
    if kind == "jobs":
        return ctx.run_jobs(st["jobs"])
    if kind == "apply":
        return st["net"].apply(st["psi"])
    if kind == "grad":
        loss, grad = st["net"].gradients(st["psi"], st["fine"])
        return {"loss": loss, "grad": grad}
    if kind == "transmission":
        return ctx.transmission(st["v"], *LATTICE, 300.0, out=st["out"])
    ax, by = cell(case)
    if kind == "ctem":
        return ctx.multislice(st["t"], st["dz"], st["seq"], ax, by, 200.0)
    if kind == "waves":
        return ctx.multislice(st["t"], st["dz"], st["seq"], ax, by, 200.0, psi=st["psi"])
    if kind == "partial":
        return ctx.partial_coherence(st["t"], st["dz"], st["seq"], ax, by, 200.0, CS, DF, 1.5, 0.0,
                                     case["mrad"] * 1e-3, df_spread=case["spread"], df_step=30.0)[0]
    if kind == "exit":
        return ctx.stem_exit_waves(st["t"], st["dz"], st["seq"], ax, by, 200.0, st["k_ap"], st["xy"], out=st["out"])
    return ctx.stem_scan(st["t"], st["dz"], st["seq"], ax, by, 200.0, st["k_ap"], st["xy"], st["det"],
                         checkpoints=st["cps"])


LATTICE = (65.248, 65.248)  # 16 cells of Au

# --------------------------------------------------------------------- work
CLOSURE_PARAMS = 75_000  # complex 3x3 layers 1 -> 32 -> ... -> 32 -> 1, real numbers
CLOSURE_FLOPS = 2 * 9 * (2 * 64 + 4 * 64 * 64 + 64 * 2)  # a pixel, forward


def _fft_flops(nx, ny):
    return 5.0 * nx * ny * math.log2(nx * ny)


def work(case):
    kind = case["kind"]
    if kind in ("apply", "grad"):
        pix = case["batch"] * case["h"] * case["w"]
        return dict(bytes=16.0 * pix + 4 * CLOSURE_PARAMS, flops=CLOSURE_FLOPS * pix * (3.0 if kind == "grad" else 1.0))
    if kind == "jobs":
        # five sides in turn, eight layers each, slices spread evenly
        sides = [(256, 384, 512, 768, 1024)[j % 5] for j in range(case["njobs"])]
        ns = (20 + case["max_slices"]) / 2.0
        return dict(bytes=sum(8.0 * n * n * (8 + 1) for n in sides),
                    flops=sum(ns * (2 * _fft_flops(n, n) + 20.0 * n * n) for n in sides))
    nx, ny = case["nx"], case["ny"]
    n2 = float(nx * ny)
    if kind == "fft":
        return dict(bytes=16.0 * n2 * case["batch"], flops=case["batch"] * _fft_flops(nx, ny))
    if kind == "potential":
        per = {"si": (5.431, 2), "srtio3": (3.905, 2.5), "au": (4.078, 2)}[case["crystal"]]
        atoms = case["cells"] ** 2 * per[1]  # of one slice
        pairs = atoms * math.pi * case["radius"] ** 2 / (case["cells"] * per[0]) ** 2 * n2
        return dict(bytes=case["nslice"] * (4.0 * n2 + 28 * atoms), flops=case["nslice"] * pairs * 12.0)
    if kind == "transmission":
        return dict(bytes=12.0 * n2 * case["nlayer"], flops=case["nlayer"] * (2 * _fft_flops(nx, ny) + 20 * n2))
    waves = case.get("nprobe", case.get("batch", 1))
    slice_flops = 2 * _fft_flops(nx, ny) + 20 * n2
    trans = 8.0 * n2 * min(case["nslice"], 16)
    if kind == "partial":
        ax, by = cell(case)
        k = case["mrad"] * 1e-3 / wavelength(200.0)
        angles = max(1.0, math.pi * k * k * ax * by)
        ndf = 2 * int(2.5 * case["spread"] / 30.0) + 1
        return dict(bytes=trans + 8.0 * n2, flops=angles * (case["nslice"] * slice_flops + ndf * _fft_flops(nx, ny)))
    out = 8.0 * waves * case["ncheck"] * case["ndet"] if kind == "stem" else 8.0 * n2 * waves
    return dict(bytes=trans + out + (8.0 * n2 * waves if kind == "waves" else 0.0),
                flops=waves * case["nslice"] * slice_flops)


# -------------------------------------------------------------------- exact
def wavelength(kev):
    return 12.3984244 / math.sqrt(kev * (2.0 * 510.99906 + kev))


def sigma_kv(kev):
    """Interaction constant in rad / (kV A)."""
    return 2.0 * math.pi * (510.99906 + kev) / (2.0 * 510.99906 + kev) / (wavelength(kev) * kev)


def _freq(n, a):
    """Spatial frequencies in float, as the program the library follows forms them."""
    i = torch.arange(n, device=DEV)
    return torch.where(i > int(n / 2.0 + 0.5), i - n, i).float() / torch.tensor(a, device=DEV).float()


def _band(nx, ny, ax, by):
    kx, ky = _freq(nx, ax), _freq(ny, by)
    f = np.float32
    k = min(f(nx) / (f(2) * f(ax)), f(ny) / (f(2) * f(by)))
    k = f(2.0 / 3.0) * k
    return (kx * kx)[:, None] + (ky * ky)[None, :] < float(f(k * k))


def _propagator(nx, ny, ax, by, kev, dz):
    kx, ky = _freq(nx, ax).double(), _freq(ny, by).double()
    a = math.pi * wavelength(kev) * dz
    return torch.exp(-1j * a * kx * kx)[:, None] * torch.exp(-1j * a * ky * ky)[None, :] * _band(nx, ny, ax, by)


def _fwd(w):
    return torch.fft.ifft2(w, norm="forward")  # exp(+i), unscaled


def _inv(w):
    return torch.fft.fft2(w, norm="forward")  # exp(-i), 1 / (nx ny)


def _slices(w, t, props, seq):
    """Spectra after the last slice's propagator."""
    for i, l in enumerate(seq):
        w = _fwd(w * t[l].to(torch.complex128)) * props[l]
        if i + 1 < len(seq):
            w = _inv(w)
    return w


def _probes(case, st, xy):
    """Waves of unit reciprocal-space amplitude inside the aperture, at positions xy."""
    ax, by = cell(case)
    nx, ny = case["nx"], case["ny"]
    ix, iy = torch.arange(nx, device=DEV), torch.arange(ny, device=DEV)
    sx = torch.where(ix < nx // 2, ix, ix - nx).double()
    sy = torch.where(iy < ny // 2, iy, iy - ny).double()
    s = ((sx / ax) ** 2)[:, None] + ((sy / by) ** 2)[None, :]
    ap = (s <= st["k_ap"] ** 2).double() / (nx * ny)
    xy = torch.as_tensor(xy, device=DEV)
    ex = torch.exp(2j * math.pi * sx[None] * (xy[:, :1] / ax))
    ey = torch.exp(2j * math.pi * sy[None] * (xy[:, 1:] / by))
    return _inv(ap * ex[:, :, None] * ey[:, None, :]) * (nx * ny), s


def _atom_potential(fp, r):
    """The library's atomic form: three K0 terms and three Gaussians."""
    v = torch.zeros_like(r)
    for i in range(3):
        a, b, c, d = fp[2 * i], fp[2 * i + 1], fp[6 + 2 * i], fp[7 + 2 * i]
        x = 2.0 * 3.141592654 * math.sqrt(b) * r
        q = (x / 3.75) ** 2
        i0 = _poly((1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813), q)
        y = x * x / 4.0
        low = -torch.log(x / 2.0) * i0 + _poly((-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698,
                                                0.00010750, 0.00000740), y)
        high = torch.exp(-x) / torch.sqrt(x) * _poly((1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872,
                                                      -0.00251540, 0.00053208), 2.0 / x)
        v += 300.8242834 * a * torch.where(x <= 2.0, low, high)
        v += 150.4121417 * c / d * torch.exp(-(3.141592654 * r) ** 2 / d)
    return v


def _poly(c, x):
    s = torch.full_like(x, c[-1])
    for v in c[-2::-1]:
        s = s * x + v
    return s


def _exact_potential(case, seed):
    spec = crystal(case, seed)
    nx, ny, ns, rad = case["nx"], case["ny"], case["nslice"], case["radius"]
    fparams = np.load(os.path.join(DATA, "fparams.npy"))
    dx, dy = spec.ax / nx, spec.by / ny
    v = torch.zeros(ns * nx * ny, dtype=torch.float64, device=DEV)
    k = np.floor(spec.z / (spec.cz / ns)).astype(np.int64)
    inside = (spec.z >= 0) & (k >= 0) & (k < ns)
    px = torch.arange(-int(rad / dx) - 2, int(rad / dx) + 3, device=DEV)
    py = torch.arange(-int(rad / dy) - 2, int(rad / dy) + 3, device=DEV)
    step = max(1, 20_000_000 // (len(px) * len(py)))
    for z in np.unique(spec.Z):
        sel = np.nonzero(inside & (spec.Z == z))[0]
        for i in range(0, len(sel), step):
            s = sel[i:i + step]
            x, y = (torch.as_tensor(q[s] % a, device=DEV) for q, a in ((spec.x, spec.ax), (spec.y, spec.by)))
            jx = torch.floor(x / dx + 0.5).long()[:, None] + px
            jy = torch.floor(y / dy + 0.5).long()[:, None] + py
            r = torch.sqrt((jx * dx - x[:, None])[:, :, None] ** 2 + (jy * dy - y[:, None])[:, None, :] ** 2)
            val = _atom_potential(fparams[z], r.clamp(min=1e-10)) * (r < rad)
            row = torch.as_tensor(k[s], device=DEV)[:, None] * nx + jx % nx
            at = row[:, :, None] * ny + (jy % ny)[:, None, :]
            v.index_add_(0, at.reshape(-1), val.reshape(-1))
    return v.view(ns, nx, ny)


def _exact_partial(case, st):
    ax, by = cell(case)
    nx, ny = case["nx"], case["ny"]
    f = np.float32
    wl, amax = f(wavelength(200.0)), f(case["mrad"] * 1e-3)
    rx, ry = f(1) / f(ax), f(1) / f(by)
    q2max = (amax / wl) * (amax / wl)
    n1, n2 = int(amax / (wl * rx) + f(1.5)), int(amax / (wl * ry) + f(1.5))
    qs = [(f(i) * rx, f(j) * ry) for j in range(-n2, n2 + 1) for i in range(-n1, n1 + 1)]
    qs = [q for q in qs if q[0] * q[0] + q[1] * q[1] <= q2max]
    x = torch.as_tensor((np.arange(nx) * ax).astype(f) / f(nx - 1), device=DEV)
    y = torch.as_tensor((np.arange(ny) * by).astype(f) / f(ny - 1), device=DEV)
    kx, ky = _freq(nx, ax), _freq(ny, by)
    k2 = (kx * kx)[:, None] + (ky * ky)[None, :]
    inside, k2 = k2 <= float(f(1.5) * f(1.5)), k2.double()
    props = [_propagator(nx, ny, ax, by, 200.0, d) for d in st["dz"]]
    lam = wavelength(200.0)
    nd = int(2.5 * case["spread"] / 30.0)
    dfs = [(DF + j * 30.0, math.exp(-0.5 * (j * 30.0 / case["spread"]) ** 2) if nd else 1.0) for j in range(-nd, nd + 1)]
    img = torch.zeros((nx, ny), dtype=torch.float64, device=DEV)
    for qx, qy in qs:
        s = ((x * float(qx))[:, None] + (y * float(qy))[None, :]).double()
        w = torch.exp(2j * float(f(3.14159265)) * s)
        w = _slices(w, st["t"], props, st["seq"])
        for df, p in dfs:
            chi = math.pi * lam * k2 * (0.5 * CS * lam * lam * k2 - df)
            img += p * _inv(w * torch.exp(-1j * chi) * inside).abs() ** 2
    return img / (len(qs) * sum(p for _, p in dfs))


def _closure_net(params, x):
    """The closure's layers in 64 bits; x: complex [b, h, w]."""
    sizes = [(1, 32)] + [(32, 32)] * 4 + [(32, 1)]
    h, off = x[:, None], 0
    for i, (ci, co) in enumerate(sizes):
        w = params[off:off + 18 * co * ci].view(3, 3, co, ci, 2)
        off += 18 * co * ci
        b = params[off:off + 2 * co].view(co, 2)
        off += 2 * co
        wr, wi = (w[..., k].permute(2, 3, 0, 1) for k in (0, 1))
        pad = torch.nn.functional.pad(torch.cat([h.real, h.imag], 1), (1, 1, 1, 1), mode="circular")
        full = torch.cat([torch.cat([wr, -wi], 1), torch.cat([wi, wr], 1)], 0)
        y = torch.nn.functional.conv2d(pad, full, b.t().reshape(-1))
        if i < 5:
            y = torch.relu(y)
        h = torch.complex(y[:, :co], y[:, co:])
    return h[:, 0]


def _exact_closure(case, st):
    p = torch.as_tensor(np.load(os.path.join(DATA, "closure_srtio3.npy")).astype(np.float64), device=DEV)
    p.requires_grad_(case["kind"] == "grad")
    outs, loss = [], 0.0
    n = case["batch"] * case["h"] * case["w"]
    for b in range(case["batch"]):
        c = st["psi"][b:b + 1].to(torch.complex128)
        s = torch.sqrt((c.abs() ** 2).sum() / 65536.0)
        if case["kind"] == "apply":
            with torch.no_grad():
                outs.append(c + s * _closure_net(p, c / s))
            continue
        d = _closure_net(p, c / s) - (st["fine"][b:b + 1].to(torch.complex128) - c) / s
        part = (d.real ** 2 + d.imag ** 2).sum() / n
        part.backward()
        loss += float(part.detach())
    return torch.cat(outs) if case["kind"] == "apply" else {"loss": loss, "grad": p.grad.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "potential":
        if 2 * (case["radius"] / (_cell_of(case) / case["nx"]) + 2) + 1 > case["nx"] or \
                2 * (case["radius"] / (_cell_of(case) / case["ny"]) + 2) + 1 > case["ny"]:
            return None  # the cutoff nearly reaches across the cell
        return _exact_potential(case, seed)
    st = prepare(case, seed)
    torch.cuda.synchronize()
    if kind in ("apply", "grad"):
        return _exact_closure(case, st)
    if kind == "fft":
        return _fwd(st["psi"].to(torch.complex128))
    if kind == "transmission":
        band = _band(case["nx"], case["ny"], *LATTICE)
        t = torch.exp(1j * sigma_kv(300.0) * 1e-3 * st["v"].double())
        return torch.cat([_inv(_fwd(x[None]) * band) for x in t])
    if kind == "partial":
        return _exact_partial(case, st)
    if kind == "jobs":
        outs = []
        for d in st["jobs"]:
            n = d["out"].shape[0]
            prop = [_propagator(n, n, d["ax"], d["by"], d["kev"], d["dz"])] * len(d["trans"])
            if "probe" in d:
                k, x, y = d["probe"]
                i = torch.arange(n, device=DEV)
                sx = torch.where(i < n // 2, i, i - n).double()
                s = ((sx / d["ax"]) ** 2)[:, None] + ((sx / d["by"]) ** 2)[None, :]
                w = _inv((s <= k * k) * torch.exp(2j * math.pi * sx * (x / d["ax"]))[:, None]
                         * torch.exp(2j * math.pi * sx * (y / d["by"]))[None, :])
            else:
                w = torch.ones((n, n), dtype=torch.complex128, device=DEV)
            outs.append(_inv(_slices(w, d["trans"], prop, d["layer_seq"])))
        return outs
    ax, by = cell(case)
    nx, ny = case["nx"], case["ny"]
    props = [_propagator(nx, ny, ax, by, 200.0, d) for d in st["dz"]]
    if kind == "ctem":
        w = torch.ones((1, nx, ny), dtype=torch.complex128, device=DEV)
        return _inv(_slices(w, st["t"], props, st["seq"]))
    if kind == "waves":
        return torch.cat([_inv(_slices(w[None].to(torch.complex128), st["t"], props, st["seq"])) for w in st["psi"]])
    step = max(1, (1 << 25) // (nx * ny))
    parts = []
    for i in range(0, case["nprobe"], step):
        w, s = _probes(case, st, st["xy"][i:i + step])
        if kind == "exit":
            parts.append(_inv(_slices(w, st["t"], props, st["seq"])))
            continue
        sums, done = [], 0
        for cp in st["cps"]:
            w = _slices(w, st["t"], props, st["seq"][done:cp + 1])
            p = w.abs() ** 2
            sums.append(torch.stack([(p * ((s >= a * a) & (s <= b * b))).sum((1, 2)) for a, b in st["det"]], 1))
            w, done = _inv(w), cp + 1
        parts.append(torch.stack(sums, 1))
    return torch.cat(parts)


def _cell_of(case):
    return case["cells"] * {"si": 5.431, "srtio3": 3.905, "au": 4.078}[case["crystal"]]
