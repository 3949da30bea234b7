"""The work a user of this framework has it do, as cases that can be timed and compared: likelihood batches of the
GLOBAL and BAYESIAN fits (Monte-Carlo and ANALYTIC models, thin and thick disks, with and without the recomputed
density profile), a CLASSIC ring fit, one model cube, a batch of different galaxies, the wind models and the
sampler's surrogate network. Sizes are those of ``bbarolo2_gb300.configs`` and ``bench.py`` and the ranges around
them.

Every input is made here from the seed, without the framework's kernels: the mock data are the analytic disk below
(or random clouds of the wind) plus noise. ``exact`` is the same disk in float64 torch, with the reference's vertical
grid and tabulated normal CDF, its FFT convolution and the log-likelihood's formula.
"""

import math

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
PIX = 8.0                                  # arcsec, of every disk case
RING_KEYS = ("radii", "xpos", "ypos", "vsys", "vrot", "vdisp", "vrad", "vvert", "dvdz", "zcyl", "dens", "z0", "inc",
             "phi", "z0thick", "fthick", "vdispthick")


def listed():
    return [
        # one likelihood of a small cube: a simplex or a line search asks for them one at a time (latency, launches)
        dict(name="point64", kind="points", model="ANALYTIC", nx=64, ny=64, nz=64, rings=16, z0=0.0, bmaj=3.0,
             bmin=3.0, nb=1, profile=False),
        # a CLASSIC fit of eight rings, VROT and VDISP free: hundreds of single-ring models, convolutions and norms
        dict(name="classic64", kind="classic", nx=64, ny=64, nz=64, rings=8, bmaj=3.0, bmin=3.0),
        # one convolved model cube handed back to the host: what a user plots or writes at the end of a fit
        dict(name="cube160", kind="cube", model="ANALYTIC", nx=160, ny=160, nz=128, rings=40, z0=1.25, bmaj=3.75,
             bmin=2.5),
        # a gradient of GLOBAL with the Monte-Carlo model: base point and 160 steps, the profile recomputed each time
        dict(name="gradient160_mc", kind="gradient", model="MC", nx=160, ny=160, nz=128, rings=40, z0=1.25,
             bmaj=3.75, bmin=2.5, nb=161, profile=True),
        # the same gradient with the ANALYTIC model (GLOBAL's default) of a thick disk
        dict(name="gradient160_an", kind="gradient", model="ANALYTIC", nx=160, ny=160, nz=128, rings=40, z0=1.25,
             bmaj=3.75, bmin=2.5, nb=161, profile=True),
        # independent points (nested sampling's proposals) with the Monte-Carlo model on an odd cube
        dict(name="points101_mc", kind="points", model="MC", nx=101, ny=97, nz=75, rings=24, z0=0.8, bmaj=4.0,
             bmin=4.0, nb=61, profile=True),
        # BAYESIAN's batch of independent points, thin ANALYTIC disk, the largest cube
        dict(name="points256_an", kind="points", model="ANALYTIC", nx=256, ny=256, nz=192, rings=20, dr=4.0, z0=0.0,
             bmaj=4.0, bmin=4.0, nb=256, profile=False),
        # a survey: galaxies of different cubes, beams and thicknesses evaluated together, four points each
        dict(name="galaxies16", kind="galaxies", ngal=16, nmin=32, nmax=200, zmax=160, nb=4),
        # WINDFIT's columns and normal equations with the shapes of the Circinus example
        dict(name="wind_circinus", kind="wind", nx=173, ny=238, nz=41, size=3.6, conelen=52.0, openang=110.0,
             bmaj=4.5, cones=1),
        # GALWIND's Monte-Carlo shells, 2.2 million clouds
        dict(name="galwind128", kind="galwind", nx=128, ny=128, nz=64, conelen=60.0, openang=60.0, cdens=20.0,
             nv=20, threads=16),
        # the surrogate network of the screened sampler: one refit and the predictions of a batch of proposals
        dict(name="refit8", kind="surrogate", dim=8, rows=16384, steps=150, batch=1024, predict=4096),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("points", "points", "points", "gradient", "gradient", "cube", "classic", "galaxies", "wind",
                       "galwind", "surrogate"))
    if kind in ("points", "gradient"):
        model = rng.choice(("MC", "ANALYTIC"))
        nx = _log(rng, 48, 200)
        c = dict(kind=kind, model=model, nx=nx, ny=nx - rng.randrange(0, 8), nz=_log(rng, 32, 160),
                 z0=round(rng.choice((0.0, rng.uniform(0.3, 1.5))), 3))
        c["rings"] = max(4, min(40, nx // 4 - rng.randrange(0, 3)))
        c["bmaj"] = round(rng.uniform(2.5, 5.0), 2)
        c["bmin"] = round(c["bmaj"] * rng.uniform(0.65, 1.0), 2)
        c["profile"] = True if kind == "gradient" else rng.choice((True, False))
        c["nb"] = min(4 * c["rings"] + 1, 161) if kind == "gradient" else _log(rng, 1, 128)
        return c
    if kind == "cube":
        nx = _log(rng, 48, 200)
        return dict(kind=kind, model="ANALYTIC", nx=nx, ny=nx - rng.randrange(0, 8), nz=_log(rng, 32, 160),
                    rings=max(4, min(40, nx // 4 - 1)), z0=round(rng.choice((0.0, rng.uniform(0.3, 1.5))), 3),
                    bmaj=round(rng.uniform(2.5, 5.0), 2), bmin=2.5)
    if kind == "classic":
        nx = rng.randrange(48, 72)
        return dict(kind=kind, nx=nx, ny=nx - rng.randrange(0, 6), nz=rng.randrange(40, 80), rings=rng.randrange(4, 9),
                    bmaj=round(rng.uniform(2.5, 4.0), 2), bmin=2.5)
    if kind == "galaxies":
        return dict(kind=kind, ngal=rng.randrange(4, 17), nmin=32, nmax=rng.randrange(80, 200),
                    zmax=rng.randrange(64, 160), nb=rng.randrange(1, 6))
    if kind == "wind":
        return dict(kind=kind, nx=rng.randrange(80, 174), ny=rng.randrange(80, 239), nz=rng.randrange(25, 48),
                    size=round(rng.uniform(3.6, 6.0), 2), conelen=round(rng.uniform(20., 52.), 1),
                    openang=round(rng.uniform(60., 110.), 1), bmaj=round(rng.uniform(3.0, 5.0), 2),
                    cones=rng.choice((1, 2)) if rng.random() < 0.3 else 1)
    if kind == "galwind":
        return dict(kind=kind, nx=rng.randrange(60, 129), ny=rng.randrange(60, 129), nz=rng.randrange(32, 80),
                    conelen=round(rng.uniform(15., 60.), 1), openang=round(rng.uniform(30., 80.), 1),
                    cdens=round(rng.uniform(5., 20.), 1), nv=rng.randrange(5, 21), threads=rng.randrange(1, 17))
    return dict(kind=kind, dim=rng.randrange(4, 45), rows=_log(rng, 1024, 32768), steps=rng.randrange(50, 151),
                batch=_log(rng, 200, 1024), predict=_log(rng, 64, 8192))


# ------------------------------------------------------------------------------------------ the disk, in float64
class _Disk:
    """The geometry of a disk case: the grid, the beam and the rings about which its points scatter."""

    def __init__(self, c, seed):
        g = np.random.default_rng([int(seed), 17])
        self.nx, self.ny, self.nz = c["nx"], c["ny"], c["nz"]
        n = min(self.nx, self.ny)
        nr = c["rings"]
        # rings every two pixels (four where the case asks), within the cube; the disk ends inside its edges
        step = c.get("dr", 2.0) if c["kind"] != "classic" else 2.0
        step = min(step, 0.5 * n / nr)
        self.step = max(step, 1.6) * PIX
        self.radii = (0.5 + np.arange(nr)) * self.step
        self.x0 = (self.nx - 1) / 2. + g.uniform(-0.4, 0.4)
        self.y0 = (self.ny - 1) / 2. + g.uniform(-0.4, 0.4)
        self.inc, self.pa = g.uniform(50., 70.), g.uniform(0., 360.)
        self.z0 = c.get("z0", 0.0) * PIX
        rmax = self.radii[-1]
        self.vrot = g.uniform(170., 210.) * (2 / math.pi) * np.arctan(self.radii / (0.1 * rmax))
        self.vdisp = np.linspace(12., 7., nr) * g.uniform(0.9, 1.1)
        self.dens = 0.8 * np.exp(-self.radii / (0.3 * rmax))
        self.vsys = 1000.
        # the line of the disk fills about 80% of the band
        self.dv = 2. * (200. * math.sin(math.radians(65.)) + 40.) / (0.8 * self.nz)
        self.ltype = 2 if self.z0 > 0 else 1
        self.bmaj, self.bmin, self.bpa = c["bmaj"] * PIX, c["bmin"] * PIX, 30.
        self.crpix3 = self.nz // 2 + 1.
        self.edges = (np.arange(self.nz + 1) + 0.5 - self.crpix3) * self.dv * 1e3 + self.vsys * 1e3      # m/s
        self.chw = self.dv * 1e3
        self.cd2i = float(np.float32(3600. / self.chw * 1000.))
        self.zstep = 0.75 if self.bmin / PIX >= 3.0 else 0.25

    def values(self):
        nr = self.radii.size
        return dict(radii=self.radii, xpos=self.x0, ypos=self.y0, vsys=self.vsys, vrot=self.vrot, vdisp=self.vdisp,
                    inc=np.full(nr, self.inc), phi=np.full(nr, self.pa), z0=np.full(nr, self.z0), dens=self.dens)

    def kernel(self):
        """The beam: a Gaussian of the FWHMs, its major axis at BPA + 90 from x, zero below 1e-4, normalised."""
        phi = math.radians(self.bpa + 90. if self.bmaj != self.bmin else 90.)
        cs, sn = math.cos(phi), math.sin(phi)
        ext = math.sqrt(math.log(1e4) / math.log(2.))
        xr, yr = 0.5 * self.bmaj * ext, 0.5 * self.bmin * ext
        hx = int(round(max(abs(xr * cs), abs(yr * sn)) / PIX))
        hy = int(round(max(abs(xr * sn), abs(yr * cs)) / PIX))
        jj, ii = np.mgrid[-hy:hy + 1, -hx:hx + 1]
        xx, yy = ii * PIX, jj * PIX
        a, b = (xx * cs + yy * sn) / self.bmaj, (-xx * sn + yy * cs) / self.bmin
        k = np.exp(-4. * math.log(2.) * (a * a + b * b))
        k = np.where(k >= 1e-4, k, 0.)
        return k / k.sum()

    def box(self, v, z0):
        ext = self.radii[-1] + self.step / 2. + 3 * z0
        d = int(math.ceil(ext / PIX))
        x, y = int(math.ceil(v["xpos"])), int(math.ceil(v["ypos"]))
        return [max(x - d, 0), max(y - d, 0)], [min(x + d + 1, self.nx), min(y + d + 1, self.ny)]


def _layer(ltype, x):
    if ltype == 1:
        return 0.5 * (1 + math.erf(x / math.sqrt(2.)))
    return 0.5 * (1 + math.tanh(x))


def _heights(d, R0, sep, sinc, x0, y0, z0, blo, bhi, coarse):
    """The vertical samples (in units of z0) and weights of a sub-ring; coarse: 9 equal steps (mock data)."""
    s = abs(sinc)
    if z0 <= 0 or s < 1e-6:
        return np.zeros(1), np.ones(1)
    pix = PIX / 60.
    dx = max(abs(blo[0] - 0.5 - x0), abs(bhi[0] - 0.5 - x0)) * pix
    dy = max(abs(blo[1] - 0.5 - y0), abs(bhi[1] - 0.5 - y0)) * pix
    zlim = min(5.0 if d.ltype == 1 else 7.6, (R0 + sep + math.hypot(dx, dy)) / (s * z0))
    core = 3.717 if d.ltype == 1 else 4.147
    if coarse:
        e = np.linspace(-2.5, 2.5, 10)
        c = np.array([_layer(d.ltype, x) for x in e])
        return 0.5 * (e[1:] + e[:-1]), np.diff(c) / (c[-1] - c[0])
    step = d.zstep * pix / (z0 * s)
    while True:
        nin = max(int(math.ceil(min(core, zlim) / step)), 1)
        nout = max(int(math.ceil((zlim - nin * step) / (4. * step))), 0)
        if 2 * (nin + nout) <= 1024:
            break
        step *= 1.01 * (nin + nout) / 512.
    j = np.arange(nin + nout)
    lo = np.where(j < nin, j, nin + 4 * (j - nin)) * step
    hi = np.minimum(lo + np.where(j < nin, step, 4. * step), zlim)
    w = np.array([_layer(d.ltype, b) - _layer(d.ltype, a) for a, b in zip(lo, hi)])
    z = 0.5 * (lo + hi)
    return np.r_[-z[::-1], z], np.r_[w[::-1], w]


_CDF = {}


def _cdf(t):
    """The normal CDF by linear interpolation in a table of 512 entries per unit from -6 (the reference's profile)."""
    if "t" not in _CDF:
        k = np.arange(6146)
        _CDF["t"] = torch.tensor([0.5 * math.erfc(-(-6. + x / 512.) / math.sqrt(2.)) for x in k], dtype=F64, device=DEV)
    tab = _CDF["t"]
    x = (t + 6.) * 512.
    i = x.clamp(0., 6144.).to(torch.int64)
    v = tab[i] + (x - i) * (tab[i + 1] - tab[i])
    return torch.where(x <= 0, torch.zeros_like(v), torch.where(x >= 6145., torch.ones_like(v), v))


def _subrings(d, v):
    """The sub-rings (0.75 pixel apart, values linear between the rings, the disk half a ring beyond both ends)."""
    sep = 0.75 * PIX / 60.
    R = d.radii
    w = d.step / 2.
    rin, rout = max(R[0] - w, 0.), R[-1] + w
    idx, rad = list(range(R.size)), list(R)
    if rin / 60. + sep < R[0] / 60.:
        idx, rad = [0] + idx, [rin] + rad
    if R[-1] / 60. + sep < rout / 60.:
        idx, rad = idx + [R.size - 1], rad + [rout]
    rad = np.array(rad) / 60.
    V = {k: np.broadcast_to(np.asarray(x, float), R.shape)[idx] for k, x in v.items() if k != "radii"}
    f32 = np.float32
    out = []
    r = f32(rad[0] + sep / 2.) if rad[0] != 0 else f32(sep / 2.)
    for i in range(1, rad.size):
        while r < f32(rad[i]):
            t = (float(r) - float(f32(rad[i - 1]))) / (rad[i] - rad[i - 1])
            out.append((float(r), {k: x[i - 1] + (x[i] - x[i - 1]) * t for k, x in V.items()}))
            r = f32(float(r) + sep)
    return out, sep


def _disk_model(d, v, blo, bhi, coarse=False):
    """The unsmoothed ANALYTIC model (by, bx, nz) of the ring values v in the box, float64."""
    by, bx, nz = bhi[1] - blo[1], bhi[0] - blo[0], d.nz
    out = torch.zeros(by * bx, nz, dtype=F64, device=DEV)
    edges = torch.tensor(d.edges, dtype=F64, device=DEV)
    chan = torch.arange(nz, device=DEV)
    pix = PIX / 60.
    subs, sep = _subrings(d, v)
    for R0, s in subs:
        area = 2 * math.pi * R0 * sep / pix ** 2
        naz = max(int(3 * 2 * math.pi * R0 / pix + 0.5), 16)
        sig = math.hypot(s["vdisp"] * 1e3, d.chw / (2 * math.sqrt(2 * math.log(2.))))
        K = int(5. * sig / d.chw) + 2
        inc, phi = math.radians(s["inc"]), math.radians(s["phi"])
        sinc, cinc, spa, cpa = math.sin(inc), math.cos(inc), math.sin(phi), math.cos(phi)
        zq, wq = _heights(d, R0, sep, sinc, s["xpos"], s["ypos"], s["z0"] / 60., blo, bhi, coarse)
        kr = torch.arange(2, dtype=F64, device=DEV)[:, None]
        R = torch.sqrt((R0 - 0.5 * sep) ** 2 + 2. * sep * R0 * (kr + 0.5) / 2.)
        az = 2 * math.pi * (torch.arange(naz, dtype=F64, device=DEV)[None] + 0.75 - 0.5 * kr) / naz
        ca, sa = torch.cos(az), torch.sin(az)
        x, yb = (R * ca).reshape(-1, 1), (R * sa * cinc).reshape(-1, 1)
        z = torch.tensor(zq * (s["z0"] / 60.), dtype=F64, device=DEV)[None]
        y = yb - z * sinc
        gx = torch.floor(s["xpos"] + (x * spa - y * cpa) / -pix + 0.5).to(torch.int64) - blo[0]
        gy = torch.floor(s["ypos"] + (x * cpa + y * spa) / pix + 0.5).to(torch.int64) - blo[1]
        vel = (s["vsys"] * 1e3 + s["vrot"] * 1e3 * ca * sinc).reshape(-1, 1)
        kc = torch.floor((vel - d.vsys * 1e3) / d.chw + d.crpix3 - 1 + 0.5).to(torch.int64)
        p = _cdf((edges[None] - vel) / sig)
        prof = (p[:, 1:] - p[:, :-1]).abs() * ((chan[None] - kc).abs() <= K)
        prof = prof * (s["dens"] * area * pix ** 2 / (2 * naz) * d.cd2i)
        ok = (gx >= 0) & (gx < bx) & (gy >= 0) & (gy < by)
        w = torch.tensor(wq, dtype=F64, device=DEV)[None] * ok
        at = torch.where(ok, gy * bx + gx, torch.zeros_like(gx))
        for j in range(z.shape[1]):
            out.index_add_(0, at[:, j], prof * w[:, j:j + 1])
    return out.reshape(by, bx, nz)


def _smooth(d, m):
    """The beam convolution ("same") of (by, bx, nz) by FFT, values below 1e-12 set to zero."""
    k = torch.tensor(d.kernel(), dtype=F64, device=DEV)
    sh = (m.shape[0] + k.shape[0] - 1, m.shape[1] + k.shape[1] - 1)
    f = torch.fft.rfft2(m, s=sh, dim=(0, 1)) * torch.fft.rfft2(k, s=sh)[..., None]
    r = torch.fft.irfft2(f, s=sh, dim=(0, 1))
    r = r[k.shape[0] // 2:k.shape[0] // 2 + m.shape[0], k.shape[1] // 2:k.shape[1] // 2 + m.shape[1]]
    return torch.where(r < 1e-12, torch.zeros_like(r), r)


def _mock(d, seed, noise=0.005):
    """(data (nz, ny, nx) float32, mask, sigma): the disk plus beam-correlated noise of 0.5% of the peak; the mask is
    the model above three times the noise grown by a beam and three channels."""
    full = ([0, 0], [d.nx, d.ny])
    truth = _smooth(d, _disk_model(d, d.values(), *full, coarse=True))
    sigma = noise * float(truth.max())
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n = _smooth(d, torch.randn(truth.shape, generator=g, dtype=F64, device=DEV) + 100.) - _smooth(
        d, torch.full_like(truth, 100.))
    n *= sigma / float(n.std())
    m = (truth > 3 * sigma).permute(2, 0, 1)[None, None].to(torch.float32)
    r = int(math.ceil(d.bmaj / PIX))
    m = torch.nn.functional.max_pool3d(m, (7, 2 * r + 1, 2 * r + 1), 1, (3, r, r))[0, 0] > 0
    data = (truth + n).permute(2, 0, 1).contiguous().to(torch.float32)
    return data.cpu().numpy(), m.cpu().numpy(), sigma


def _disk_cube(c, d, data=None, model="MC"):
    from bbarolo2_gb300.cube import Cube, Params
    par = Params(CDENS=10, ISEED=1, LTYPE=d.ltype, galmodtype=model)
    cube = Cube.empty(d.nx, d.ny, d.nz, [-PIX / 3600., PIX / 3600., d.dv],
                      beam=[d.bmaj / 3600., d.bmin / 3600., d.bpa if d.bmaj != d.bmin else 0.], par=par,
                      crpix=[d.nx / 2. + 0.5, d.ny / 2. + 0.5, d.crpix3], crval=[60., 0., d.vsys],
                      cunit=("deg", "deg", "km/s"))
    if data is not None:
        cube.array = data
    return cube


def _disk_rings(d):
    from bbarolo2_gb300.rings import Rings
    v = d.values()
    return Rings().setRings(**v)


def _rows(c, d, seed):
    """The ring-value rows (nb, 17, nr): a gradient's base point and steps, or independent points about it."""
    nr, nb = d.radii.size, c["nb"]
    v = d.values()
    base = np.zeros((17, nr))
    base[16] = -1.
    for k, x in v.items():
        base[RING_KEYS.index(k)] = x
    rows = np.repeat(base[None], nb, axis=0)
    g = np.random.default_rng([int(seed), 5])
    if c["kind"] == "gradient":
        k = 1
        for j in range(nr):
            for row, step in ((4, 2.0), (5, 0.5), (12, 0.5), (13, 0.5)):
                if k < nb:
                    rows[k, row, j] += step * (1 + 0.1 * g.random())
                    k += 1
        return rows
    for row, half in ((4, 5.0), (5, 1.0)):
        rows[:, row] += g.uniform(-half, half, (nb, nr))
    for row, half in ((12, 1.0), (13, 1.0)):
        rows[:, row] += g.uniform(-half, half, (nb, 1))
    return rows


# ------------------------------------------------------------------------------------------ preparing and running
def _prepare_likelihood(c, seed):
    from bbarolo2_gb300 import engine
    d = _Disk(c, seed)
    data, mask, sigma = _mock(d, seed)
    cube = _disk_cube(c, d, model=c["model"])
    rings = _disk_rings(d)
    dm = engine.DiskModel(cube, galmodtype=c["model"])
    like = engine.BatchLikelihood(dm, data, mask, maskmode=2, sigma=sigma)
    if c["profile"]:
        mom0, rms, ok = like.data_maps()
        area = math.pi * d.bmaj * d.bmin / (4. * math.log(2.)) / PIX ** 2
        like.set_profile(rings, mom0, rms, ok, smooth=0.3, corr=area, beam_arcsec=d.bmaj)
    return dict(kind="like", like=like, rings=rings, rows=_rows(c, d, seed), model=c["model"])


def _prepare_cube(c, seed):
    from bbarolo2_gb300 import engine
    d = _Disk(c, seed)
    dm = engine.DiskModel(_disk_cube(c, d, model=c["model"]), galmodtype=c["model"])
    return dict(kind="cube", dm=dm, rings=_disk_rings(d))


def _prepare_classic(c, seed):
    from bbarolo2_gb300 import classic
    d = _Disk(c, seed)
    data, mask, sigma = _mock(d, seed, noise=0.01)
    cube = _disk_cube(c, d, data)
    rings = _disk_rings(d)
    rings.vrot = np.full(rings.nr, 120.)
    rings.vdisp = np.full(rings.nr, 8.)
    return dict(kind="classic", fit=classic.ClassicFit(cube, rings, classic.default_par(), sigma, mask))


def _population(c, seed):
    """The sizes of the galaxies (of the case alone) and their values (of the seed)."""
    g, s = np.random.default_rng(11), np.random.default_rng([int(seed), 3])
    for _ in range(c["ngal"]):
        nx, nz = int(g.integers(c["nmin"], c["nmax"] + 1)), int(g.integers(32, c["zmax"] + 1))
        nr = max(min(int(g.integers(5, 51)), int(0.2 * nx)), 2)
        z0, fwhm = float(g.uniform(0., 0.2)) * 0.4 * nx, float(g.uniform(2., 6.))
        yield dict(kind="galaxy", nx=nx, ny=nx, nz=nz, rings=nr, dr=0.4 * nx / nr, z0=z0, bmaj=fwhm, bmin=fwhm,
                   nb=c["nb"], model="ANALYTIC"), int(s.integers(1 << 30))


def _prepare_galaxies(c, seed):
    from bbarolo2_gb300.ragged import GalaxyBatch
    items, rows = [], []
    for gc, s in _population(c, seed):
        d = _Disk(gc, s)
        d.ltype = 1
        data, mask, sigma = _mock(d, s, noise=0.01)
        items.append((_disk_cube(gc, d, model="ANALYTIC"), _disk_rings(d), data, mask, sigma))
        rows.append(_rows(gc, d, s))
    return dict(kind="galaxies", batch=GalaxyBatch(items), rows=rows)


def _wind_clouds(p, cube, n, seed):
    """A mock wind cube (nz, ny, nx): n random points of the cone with emissivity r^-3.4, binned and smoothed."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    u = torch.rand(3, n, generator=g, dtype=F64, device=DEV)
    r = 2.0 + u[0] * (p["conelen"] - 2.0)
    ct = 1 - u[1] * (1 - math.cos(math.radians(p["openang"] / 2)))
    st, ph = torch.sqrt(1 - ct * ct), 2 * math.pi * u[2]
    w = r ** 2 * (r / 26.) ** -3.4
    inc, pa = math.radians(p["inc"]), math.radians(p["pa"])
    z = -r * ct
    x, ys = r * st * torch.cos(ph), r * st * torch.sin(ph) * math.cos(inc) - z * math.sin(inc)
    gx = torch.round(p["xpos"] - (x * math.sin(pa) - ys * math.cos(pa)) / 0.2).to(torch.int64)
    gy = torch.round(p["ypos"] + (x * math.cos(pa) + ys * math.sin(pa)) / 0.2).to(torch.int64)
    vel = p["vwind"] * (-ct * math.cos(inc) + st * torch.sin(ph) * math.sin(inc))
    k = torch.round(vel / 75. + cube.nz * 0.56).to(torch.int64)
    ok = (gx >= 0) & (gx < cube.nx) & (gy >= 0) & (gy < cube.ny) & (k >= 0) & (k < cube.nz)
    out = torch.zeros(cube.nz * cube.ny * cube.nx, dtype=F64, device=DEV)
    out.index_add_(0, ((k * cube.ny + gy) * cube.nx + gx)[ok], w[ok])
    out = out.reshape(1, cube.nz, cube.ny, cube.nx)
    e = torch.exp(-0.5 * (torch.arange(-6, 7, dtype=F64, device=DEV) / 2.) ** 2)
    e = e / e.sum()
    f = torch.nn.functional.conv2d(out[0][:, None], e[None, None, :, None], padding=(6, 0))
    f = torch.nn.functional.conv2d(f, e[None, None, None, :], padding=(0, 6))[:, 0]
    f = f + 0.3 * torch.roll(f, 1, 0) + 0.3 * torch.roll(f, -1, 0)
    return f


def _prepare_wind(c, seed):
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.wind import WindCells, WindModel, WindPars
    g = np.random.default_rng([int(seed), 9])
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    crpix3 = float(round(nz * 0.56) + 1)
    cube = Cube.empty(nx, ny, nz, [-0.2 / 3600., 0.2 / 3600., 75.], beam=0.2 * c["bmaj"] / 3600.,
                      par=Params(specres=0.85), crpix=[nx / 2. + 0.5, ny / 2. + 0.5, crpix3], crval=[213.29, -65.34, 0.],
                      cunit=("deg", "deg", "km/s"))
    cells = WindCells.resolved(c["conelen"], c["openang"] / 2., c["size"], cones=(-1,) if c["cones"] == 1 else (1, -1))
    wm = WindModel(cube, cells).quadrature(vmax=1600., sigmin=0.)
    p = dict(xpos=0.115 * nx + g.uniform(-1, 1), ypos=0.17 * ny + g.uniform(-1, 1), inc=71.6 + g.uniform(-1, 1),
             pa=25. + g.uniform(-2, 2), openang=c["openang"], conelen=c["conelen"], vwind=338. + g.uniform(-20, 20))

    class Dim:
        pass
    dim = Dim()
    dim.nx, dim.ny, dim.nz = nx, ny, nz
    m = _wind_clouds(p, dim, 2_000_000, seed)
    peak = float(m.max())
    sig = 0.05 * peak
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    data = m + sig * torch.randn(m.shape, generator=gen, dtype=F64, device=DEV)
    W = torch.where(m > 1e-3 * peak, 1. / sig ** 2, 0. * m)
    wp = WindPars([c["conelen"] / 2], p["vwind"], 0., xpos=p["xpos"], ypos=p["ypos"], inc=p["inc"], pa=p["pa"],
                  openang=p["openang"], conelen=p["conelen"])
    return dict(kind="wind", wm=wm, p=wp, W=W.cpu().numpy(), Wd=(W * data).cpu().numpy())


def _prepare_galwind(c, seed):
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galwind import GalWindMC, GalWindPars
    g = np.random.default_rng([int(seed), 21])
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    cube = Cube.empty(nx, ny, nz, [-4. / 3600., 4. / 3600., 640. / nz], par=Params(),
                      crpix=[nx / 2. + 0.5, ny / 2. + 0.5, nz / 2. + 0.5], crval=[60., 0., 0.],
                      cunit=("deg", "deg", "km/s"))
    # CONELEN in pixels of 4", shells of 30 layers (fewer for a short cone: a layer spans two pixels)
    par = GalWindPars(xpos=(nx - 1) / 2. + g.uniform(-1, 1), ypos=(ny - 1) / 2. + g.uniform(-1, 1), vsys=0.,
                      inc=60. + g.uniform(-5, 5), phi=g.uniform(0., 360.), conelen=4. * c["conelen"],
                      nlayers=max(3, min(30, int(c["conelen"] / 2.))), vwind=300., vdisp=20., dens=10.,
                      openang=c["openang"], cdens=c["cdens"], nv=c["nv"], iseed=int(g.integers(1, 1 << 20)))
    return dict(kind="galwind", wind=GalWindMC(cube, par, threads=c["threads"]))


def _prepare_surrogate(c, seed):
    from bbarolo2_gb300.surrogate import MLP
    g = np.random.default_rng([int(seed), 33])
    x = g.standard_normal((c["rows"], c["dim"])).astype(np.float32)
    t = np.clip(1. - 0.5 * (x * x).sum(axis=1) / c["dim"] + 0.05 * g.standard_normal(c["rows"]), -1, 1)
    net = MLP(c["dim"], 256, seed=int(seed) % 1000)
    return dict(kind="surrogate", net=net, p0=net.params(), x=x, t=t.astype(np.float32),
                q=g.standard_normal((c["predict"], c["dim"])).astype(np.float32), steps=c["steps"],
                batch=min(c["batch"], c["rows"]))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("points", "gradient"):
        return _prepare_likelihood(case, seed)
    return {"cube": _prepare_cube, "classic": _prepare_classic, "galaxies": _prepare_galaxies, "wind": _prepare_wind,
            "galwind": _prepare_galwind, "surrogate": _prepare_surrogate}[kind](case, seed)


def run(s):
    kind = s["kind"]
    if kind == "like":
        return s["like"].evaluate(s["rows"], s["rings"], seed=1, galmodtype=s["model"])
    if kind == "cube":
        return s["dm"].array(s["rings"], seed=1)
    if kind == "classic":
        out, ok = s["fit"].run()
        return out.vrot, out.vdisp, [bool(v) for v in ok], [float(s["fit"].status[i][1]) for i in range(out.nr)]
    if kind == "galaxies":
        return s["batch"].evaluate(s["rows"], seed=1)
    if kind == "wind":
        B = s["wm"].boxes(s["p"])
        return B.normal(s["Wd"], s["W"], B.voxel_lists(s["W"], rel=1e-3))
    if kind == "galwind":
        return s["wind"].model()
    # (a refit from the same weights each time, so that a pass can be repeated)
    s["net"].set_params(s["p0"])
    loss = s["net"].train(s["x"], s["t"], s["steps"], s["batch"], seed=7)
    return s["net"].params(), loss, s["net"].predict(s["q"])


# ------------------------------------------------------------------------------------------ the work and the truth
def _disk_work(c, seed=1):
    """Least bytes and operations of a disk batch: the rows, the data and mask of the box read, the result written;
    per member the deposits (3 operations a value), the convolution (2 a non-zero tap and voxel) and the residual."""
    d = _Disk(c, seed)
    v = d.values()
    blo, bhi = d.box(v, d.z0)
    vox = (bhi[0] - blo[0]) * (bhi[1] - blo[1]) * d.nz
    nb = c.get("nb", 1)
    pix = PIX / 60.
    per = 0.
    for R0, s in _subrings(d, v)[0]:
        K = int(5. * math.hypot(s["vdisp"] * 1e3, d.chw / 2.3548) / d.chw) + 2
        if c.get("model") == "MC":
            per += 10 * 2 * math.pi * R0 * 0.75 / pix * d.nz * 8       # 10 clouds a pixel, NV = the channels
        else:
            per += 2 * 3 * 2 * math.pi * R0 / pix * (2 * K + 1) * 3 * (1 if d.z0 <= 0 else 4)
    taps = int(np.count_nonzero(d.kernel()))
    rows = 17 * d.radii.size * 8
    return vox, nb, nb * (per + vox * (2 * taps + 3)), vox * 5 + nb * (rows + 8)


def work(case):
    kind = case["kind"]
    if kind in ("points", "gradient"):
        _, _, flops, nbytes = _disk_work(case)
        return {"bytes": nbytes, "flops": flops}
    if kind == "cube":
        _, _, flops, nbytes = _disk_work(case)
        return {"bytes": nbytes + 8 * case["nx"] * case["ny"] * case["nz"], "flops": flops}
    if kind == "classic":
        # about 40 evaluations a ring of a box that the ring fills
        d = _Disk(case, 1)
        vox = sum(40 * (2 * r / PIX + 6) ** 2 * d.nz for r in d.radii)
        return {"bytes": case["nx"] * case["ny"] * case["nz"] * 5, "flops": vox * 2 * np.count_nonzero(d.kernel()) * 0.3}
    if kind == "galaxies":
        b = f = 0
        for gc, _ in _population(case, 1):
            _, _, flops, nbytes = _disk_work(gc)
            b, f = b + nbytes, f + flops
        return {"bytes": b, "flops": f}
    if kind == "wind":
        # the cells' sizes over the cone's volume, 600 points of 12 channels x 4 pixels each, the columns' convolution
        n = _wind_cells(case)
        side = case["size"] / 0.2 + 4 * case["bmaj"]
        col = side * side * 8
        return {"bytes": 16 * case["nx"] * case["ny"] * case["nz"] + 8 * n * n,
                "flops": n * (600 * 12 * 10 + col * 4 * 4 * case["bmaj"] + col * 20)}
    if kind == "galwind":
        n, nv = _galwind_clouds(case), case["nv"]
        return {"bytes": 8 * case["nx"] * case["ny"] * case["nz"], "flops": n * (60 + nv * 20)}
    np_ = case["dim"] * 256 + 2 * 256 * 256 + 256
    return {"bytes": 4 * (case["rows"] * (case["dim"] + 1) + 2 * np_ + case["predict"] * (case["dim"] + 1)),
            "flops": case["steps"] * (6 * np_ * min(case["batch"], case["rows"]) + 12 * np_) + 2 * np_ * case["predict"]}


def _wind_cells(c):
    v = 2 * math.pi / 3 * c["conelen"] ** 3 * (1 - math.cos(math.radians(c["openang"] / 2)))
    return c["cones"] * v / c["size"] ** 3


def _galwind_clouds(c):
    r = np.arange(0.375, c["conelen"], 0.75)
    return float(np.sum(c["cdens"] * 10. * 2 * math.pi * r * 0.75))


def exact(case, seed):
    """float64 values of the ANALYTIC disks: the model cube, or log L of every point. None: the Monte-Carlo models
    (their clouds are a sequential random stream of tens of millions of draws), the fits and the surrogate (hundreds
    of evaluations or steps), the wind's normal equations and the gradients (a constrained least squares a member, or
    thousands of boxes each with its selection): each beyond some 20 seconds of plain torch."""
    kind = case["kind"]
    if kind == "cube":
        d = _Disk(case, seed)
        m = _smooth(d, _disk_model(d, d.values(), [0, 0], [d.nx, d.ny]))
        return m.permute(2, 0, 1).contiguous()
    if kind != "points" or case["model"] != "ANALYTIC" or case["profile"]:
        return None
    if _exact_cost(case) > 1e12:
        return None
    d = _Disk(case, seed)
    data, mask, sigma = _mock(d, seed)
    D = torch.tensor(data, device=DEV).to(F64).permute(1, 2, 0)
    ok = torch.tensor(mask, device=DEV).permute(1, 2, 0) & (D != 0)
    total = float((D * D)[ok].sum())
    out = []
    for row in _rows(case, d, seed):
        v = {k: row[RING_KEYS.index(k)] for k in ("vrot", "vdisp", "inc", "phi", "z0", "dens", "vsys")}
        v.update(xpos=d.x0, ypos=d.y0)
        blo, bhi = d.box(dict(xpos=d.x0, ypos=d.y0), d.z0)
        m = _smooth(d, _disk_model(d, v, blo, bhi))
        sl = (slice(blo[1], bhi[1]), slice(blo[0], bhi[0]))
        inside = ok[sl]
        ss = float(((D[sl] - m)[inside] ** 2).sum()) + max(total - float((D[sl][inside] ** 2).sum()), 0.)
        out.append(-(0.5 * ss / sigma ** 2 + 0.5 * int(ok.sum()) * math.log(2 * math.pi * sigma ** 2)))
    return np.array(out)


def _exact_cost(c):
    """Operations of the plain float64 model of every point (samples x heights x channels)."""
    d = _Disk(c, 1)
    heights = 1 if d.z0 <= 0 else 2 * math.ceil(4.2 * d.z0 / (d.zstep * PIX))
    return c["nb"] * sum(2 * 3 * 2 * math.pi * r / (PIX / 60.) for r, _ in _subrings(d, d.values())[0]) * d.nz * (
        40 + 4 * heights)
