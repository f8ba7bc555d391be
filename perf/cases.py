"""Performance cases of the multislice ADF-STEM / FEM library.

Each case is work a user has the library do through its Python binding
(`msf.py`, one call per C ABI entry point): a raster over a resident specimen,
a specimen build followed by its raster, several uneven rasters in one call,
an MD-averaged raster, and a burst of requests to the serving loop.  Grids
sample the cell at 100 A / 1024 per pixel and slices are 2 A, as in the
benchmark workloads; specimens are seeded amorphous-like Si (or Si and O) at
50 atoms per nm^3.

`exact` restates the same simulation in FP64 with torch FFTs and numpy and
uses none of the library.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ms-stem-fem_b200"))
import msf  # noqa: E402

SAMPLING = 100.0 / 1024.0   # A per pixel
DENSITY = 0.05              # atoms per A^3
MIN_SLICE = 2.0             # A
DET_INNER, DET_OUTER = 0.04, 0.2  # rad
MODES = ("V_omega", "Vbar_r", "V_re", "Omega_vimage", "V_gt17", "V_rbar")
# detector MTF table (domain in Nyquist units, value) and its sampling rate
MTF_DOMAIN = (0.0, 0.25, 0.5, 0.75, 1.0, 1.5)
MTF_VALUE = (1.0, 0.8, 0.55, 0.35, 0.2, 0.1)
MTF_RATE = 20.0


def _case(name, kind, nx, ny, precision, depth, rx, ry, **more):
    """kind: run, build, batch, md or serve; depth [A]; rx x ry probes.
    optics: "fem" (1.5 mrad, in focus), "adf" (10 mrad, Scherzer defocus),
    "corrected" (Cs5-corrected Scherzer).  outputs: "adf" or FEM mode names
    joined by "+" (the ADF image is always returned)."""
    c = dict(kind=kind, nx=nx, ny=ny, precision=precision, depth=depth, rx=rx, ry=ry,
             voltage=200000.0, optics="adf", outputs="adf", oxide=False, mtf=False,
             waves=False, samples=1, snapshots=1, jobs=1)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest job of the examples: a few probes on a tiny cell, where
        # launches and host steps count; also writes diffraction images
        _case("fem_128x64_fp32", "run", 128, 64, "fp32", 25.0, 4, 4,
              outputs="V_omega+Vbar_r", waves=True),
        # a quick ADF image in the library's default precision
        _case("adf_256_fp64", "run", 256, 256, "fp64", 12.0, 8, 8, waves=True),
        # a burst of small requests to the serving loop
        _case("serve_256_512_fp32", "serve", 256, 256, "fp32", 14.0, 6, 7,
              outputs="V_omega", jobs=6),
        # thermal / MD averaging: 2 configurations, 4 samples per probe
        _case("md_256_fp32", "md", 256, 256, "fp32", 10.0, 6, 6,
              outputs="+".join(MODES), samples=4, snapshots=2),
        # an aberration-corrected probe on an odd raster
        _case("fem_512_corrected_fp32", "run", 512, 512, "fp32", 11.0, 13, 11,
              optics="corrected", outputs="V_omega"),
        # a rectangular oxide cell with the detector MTF before the FEM sums
        _case("fem_512x256_mtf_fp32", "run", 512, 256, "fp32", 15.0, 7, 5, oxide=True,
              mtf=True, outputs="V_omega+V_re+Omega_vimage"),
        # uneven specimens sharing launches (one lane per grid size)
        _case("batch_256_1024_fp32", "batch", 512, 512, "fp32", 24.0, 9, 10, optics="fem",
              outputs="V_omega", jobs=4),
        # the FP64 check of an FEM specimen
        _case("fem_1024_fp64", "run", 1024, 1024, "fp64", 20.0, 8, 8,
              outputs="V_omega+V_re"),
        # a new specimen from host atoms, then its raster
        _case("build_fem_1024_fp32", "build", 1024, 1024, "fp32", 100.0, 6, 6, optics="fem",
              outputs="V_omega+V_re"),
        # the FEM variance raster the benchmark is quoted on, 16 x 16 of its
        # 64 x 64 probes
        _case("fem_1024_fp32", "run", 1024, 1024, "fp32", 100.0, 16, 16, optics="fem",
              outputs="V_omega+V_re"),
        # a large field of view at 300 kV
        _case("adf_2048_fp32", "run", 2048, 2048, "fp32", 100.0, 5, 5, voltage=300000.0,
              outputs="V_omega"),
        # the largest grid
        _case("adf_4096_fp32", "run", 4096, 4096, "fp32", 10.0, 2, 3, voltage=300000.0),
    ]


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["build", "batch", "md", "serve"])
    precision = "fp64" if kind in ("run", "build") and rng.random() < 0.3 else "fp32"
    sides = (64, 128, 256, 512, 1024, 2048, 4096) if kind in ("run", "build") else (128, 256, 512)
    nx = rng.choice(sides)
    ny = nx if rng.random() < 0.6 else max(64, nx // rng.choice((2, 4)))
    if rng.random() < 0.3:
        nx, ny = ny, nx
    depth = round(math.exp(rng.uniform(math.log(4.0), math.log(100.0))), 1)
    # probe*slice*pixels at most those of the largest listed case (FP64 costs
    # about three times as much), specimens at most as large as its own
    plane = nx * ny
    most = 256 * 50 * 1024 * 1024 / (3.0 if precision == "fp64" else 1.0)
    most /= 6.0 if kind in ("batch", "md", "serve") else 1.0
    depth = min(depth, max(4.0, round(100.0 * 1024 * 1024 / plane, 1)))
    probes = min(1000.0 if kind in ("run", "build") else 250.0, most / (plane * depth / 2.0))
    n = math.exp(rng.uniform(0.0, math.log(max(2.0, probes))))
    rx = max(1, int(round(math.sqrt(n) * rng.uniform(0.7, 1.4))))
    ry = max(1, int(n / rx))
    # an in-focus 1.5 mrad probe needs a large cell, and leaves the rings of an
    # FP64 raster at the rounding of its direct beam, with no figure to compare
    optics = rng.choice(("adf", "fem", "corrected")) if min(nx, ny) >= 512 else "adf"
    if optics == "fem" and precision == "fp64":
        optics = "adf"
    modes = [m for m in MODES if rng.random() < 0.4]
    mtf = kind == "run" and bool(modes) and plane <= 512 * 512 and rng.random() < 0.3
    return _case(None, kind, nx, ny, precision, depth, rx, ry,
                 voltage=rng.choice((100000.0, 200000.0, 300000.0)), optics=optics,
                 outputs="+".join(modes) or "adf", oxide=rng.random() < 0.3, mtf=mtf,
                 waves=kind == "run" and plane <= 512 * 512 and rng.random() < 0.5,
                 samples=4 if kind == "md" else 1, snapshots=2 if kind == "md" else 1,
                 jobs=rng.randint(2, 5) if kind in ("batch", "serve") else 1)


# ------------------------------------------------------------------ inputs --
def _rasters(case):
    """The case's simulations: one, or (batch, serve) several uneven ones
    around its size."""
    if case["jobs"] == 1:
        return [case]
    out = []
    for k in range(case["jobs"]):
        f = (1, 1, 2, 0.5, 1, 1)[k % 6]
        out.append(dict(case, nx=max(64, int(case["nx"] * f)), ny=max(64, int(case["ny"] * f)),
                        rx=max(1, case["rx"] - k % 3), ry=case["ry"] + (k % 2),
                        depth=case["depth"] * (1.0 + 0.1 * k)))
    return out


def _atoms(case, seed):
    """Positions [n, 3] and atomic numbers: one atom per cell of a lattice of
    the target density, jittered in x and y, uniform in z within its cell."""
    rng = np.random.default_rng(seed)
    box = np.array([case["nx"] * SAMPLING, case["ny"] * SAMPLING, case["depth"]])
    n = np.maximum(1, np.round(box * DENSITY ** (1.0 / 3.0))).astype(int)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    jitter = np.stack([rng.uniform(0.4, 0.6, len(g)), rng.uniform(0.4, 0.6, len(g)),
                       rng.uniform(0.0, 1.0, len(g))], 1)
    q = (g + jitter) * (box / n)
    z = np.full(len(q), 14, np.uint32)
    if case["oxide"]:
        z[rng.random(len(q)) < 2.0 / 3.0] = 8
    return np.ascontiguousarray(q[rng.permutation(len(q))]), z


def _raster_points(case):
    return (np.arange(case["rx"]) * (case["nx"] * SAMPLING / case["rx"]),
            np.arange(case["ry"]) * (case["ny"] * SAMPLING / case["ry"]))


def _modes(case):
    return [m for m in case["outputs"].split("+") if m in MODES]


def _wavelength(voltage):
    """Electron wavelength [A] and interaction factor, with the constants of
    the program."""
    m, c, e, h = 9.109e-31, 299792458.0, 1.60217662e-19, 6.62607004e-34
    rest, ev = m * c * c, e * voltage
    lam = h * c * 1e10 / math.sqrt(ev * (2.0 * rest + ev))
    gam = (h * 1e10 / lam) ** 2 * (rest + ev) / ((2 * rest + ev) * ev * m)
    return lam, gam


def _optics(case):
    """corrected, cs3, cs5, defocus, alpha_max"""
    lam = _wavelength(case["voltage"])[0]
    if case["optics"] == "fem":
        return 0, 1.3e7, 0.0, 0.0, 0.0015
    if case["optics"] == "adf":
        return 0, 1.3e7, 0.0, 0.87 * math.sqrt(1.3e7 * lam), 0.010
    cs5 = 5e7
    return (1, -2.289 * (lam * cs5 ** 2) ** (1.0 / 3.0), cs5,
            -0.983 * (lam ** 2 * cs5) ** (1.0 / 3.0), 1.513 * (lam / cs5) ** (1.0 / 6.0))


def _structs(case):
    """The call's argument structs and the arrays they point to."""
    keep = []

    def ptr(a):
        a = np.ascontiguousarray(a, np.float64)
        keep.append(a)
        return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))

    grid = msf.Grid(nx=case["nx"], ny=case["ny"], voltage=case["voltage"],
                    xperiod=case["nx"] * SAMPLING, yperiod=case["ny"] * SAMPLING,
                    zperiod=case["depth"], dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0,
                    xmin=0.0, ymin=0.0, zmin=0.0, min_slice=MIN_SLICE)
    xp, yp = _raster_points(case)
    raster = msf.Raster(len(xp), len(yp), ptr(xp), ptr(yp))
    outputs = msf.OUT_ADF_IMAGE
    for m in _modes(case):
        outputs |= msf.FEM_MODES[m]
    detect = msf.Detect(outputs=outputs, det_inner=DET_INNER, det_outer=DET_OUTER, dr=1.2065)
    if case["mtf"]:
        detect.n_mtf = len(MTF_VALUE)
        detect.mtf = ptr(MTF_VALUE)
        detect.mtf_domain_sqr = ptr((0.5 * MTF_RATE * np.array(MTF_DOMAIN)) ** 2)
        detect.mtf_resolution = MTF_RATE
    return grid, msf.Optics(*_optics(case)), raster, detect, keep


def _snapshot_atoms(case, seed):
    """The MD configurations of a case: one specimen, thermally displaced."""
    q, z = _atoms(case, seed)
    box = np.array([case["nx"] * SAMPLING, case["ny"] * SAMPLING])
    out = [(q, z)]
    for k in range(1, case["snapshots"]):
        p = q + np.random.default_rng([seed, k]).normal(0.0, 0.08, q.shape)
        p[:, :2] %= box
        p[:, 2] = np.clip(p[:, 2], 0.0, case["depth"])
        out.append((p, z))
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "kind": kind, "jobs": []}
    if kind == "serve":  # a running server; each request brings its specimen
        state["server"] = msf.Server()
    else:
        state["ctx"] = msf.Context(precision=case["precision"])
    for k, c in enumerate(_rasters(case)):
        grid, optics, raster, detect, keep = _structs(c)
        job = {"case": c, "grid": grid, "optics": optics, "raster": raster, "detect": detect,
               "keep": keep, "atoms": _snapshot_atoms(c, 1000 * seed + k)}
        if kind in ("run", "batch", "md"):  # resident specimens
            job["specs"] = [state["ctx"].specimen(grid, q, z) for q, z in job["atoms"]]
        state["jobs"].append(job)
    return state


def _results(case, res):
    """What the raster computed.  FP32 rasters carry FP32 accuracy in their
    double buffers; a program keeps them as float32."""
    keep = np.float32 if case["precision"] == "fp32" else np.float64
    out = {"adf_image": res.adf_image_2d.astype(keep), "bin_counts": res.counts}
    for m, v in res.v.items():
        out[m] = v.astype(keep)
    if case["waves"]:
        out["final_psi"] = res.final_psi_2d.astype(keep)
    return out


def run(state):
    kind, jobs, case = state["kind"], state["jobs"], state["case"]
    j = jobs[0]
    if kind == "run":
        res = state["ctx"].run(j["specs"][0], j["optics"], j["raster"], j["detect"],
                               want_final_psi=case["waves"])
        return _results(case, res)
    if kind == "build":
        spec = state["ctx"].specimen(j["grid"], *j["atoms"][0])
        res = state["ctx"].run(spec, j["optics"], j["raster"], j["detect"],
                               want_final_psi=case["waves"])
        spec.close()
        return _results(case, res)
    if kind == "md":
        res = state["ctx"].run_md(j["specs"], case["samples"], j["optics"], j["raster"],
                                  j["detect"])
        return _results(case, res)
    if kind == "batch":
        outs = state["ctx"].run_batch([(x["specs"][0], x["optics"], x["raster"], x["detect"])
                                       for x in jobs])
        return [_results(case, r) for r in outs]
    server = state["server"]
    tickets = [server.submit(x["grid"], *x["atoms"][0], x["optics"], x["raster"], x["detect"])
               for x in jobs]
    outs = []
    for t in tickets:
        res = None
        while res is None:
            res = server.poll(t, wait_ms=200)
        outs.append(_results(case, res))
    return outs


def work(case):
    """FFT and point-wise arithmetic of the slice loop; the transmission
    functions (FP32 or FP64 complex) or atoms read once, the results written."""
    flops = total = 0.0
    for c in _rasters(case):
        plane = c["nx"] * c["ny"]
        slices = max(1.0, c["depth"] / MIN_SLICE)
        flops += (c["rx"] * c["ry"] * slices * c["samples"] *
                  (10.0 * plane * math.log2(plane) + 20.0 * plane))
        cplx = 8.0 if c["precision"] == "fp32" else 16.0
        if c["kind"] in ("build", "serve"):
            total += 28.0 * DENSITY * plane * SAMPLING ** 2 * c["depth"]
        else:
            total += cplx * plane * slices * c["snapshots"]
        total += 8.0 * c["rx"] * c["ry"] + (16.0 * plane if c["waves"] else 0.0)
    return {"bytes": total, "flops": flops}


# ------------------------------------------------------- FP64 restatement --
_PI = 3.14159265369  # the program's constant
# Kirkland parameters {a, b, c, d} in the program's order, by atomic number
_KIRKLAND = {
    8: (3.39969204e-001, 3.07570172e-001, 1.30369072e-001, 3.81570280e-001, 3.81571436e-001,
        1.91919745e+001, 8.83326058e-002, 1.96586700e-001, 9.96220028e-004, 7.60635525e-001,
        2.07401094e+000, 3.03266869e-002),
    14: (1.06543892e+000, 1.20143691e-001, 1.80915263e-001, 1.04118455e+000, 6.87113368e+001,
         8.87533926e-002, 1.12065620e+000, 3.05452816e-002, 1.59963502e+000, 3.70062619e+000,
         2.14097897e-001, 9.99096638e+000),
}


def _snap(x, q, last):
    """First pixel half a step or more past q, minus one; `last` when none."""
    hit = np.nonzero(x - q >= 0.5 * (x[1] - x[0]))[0]
    return int(hit[0]) - 1 if len(hit) else last


def _slices(q):
    """Atom index lists and thicknesses: a slice takes the atoms within
    MIN_SLICE above its lowest one and lies at their mean height."""
    order = np.argsort(q[:, 2], kind="stable")
    zs = q[order, 2]
    start = [0]
    while True:
        k = start[-1] + int(np.searchsorted(zs[start[-1]:] - zs[start[-1]], MIN_SLICE, "right"))
        if k >= len(zs):
            break
        start.append(k)
    start.append(len(zs))
    lower = [zs[a:b].sum() / (b - a) for a, b in zip(start, start[1:])]
    thick = list(np.diff(lower)) + [zs[-1] + MIN_SLICE - lower[-1]]
    return [order[a:b] for a, b in zip(start, start[1:])], thick


class _Cell:
    """Grid, band limit and transforms of a case, in FP64."""

    def __init__(self, case):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny = self.nx, self.ny = case["nx"], case["ny"]
        self.lx, self.ly = nx * SAMPLING, ny * SAMPLING
        self.lam, self.gam = _wavelength(case["voltage"])
        i, j = np.arange(nx), np.arange(ny)
        self.x, self.y = i * (self.lx / nx), j * (self.ly / ny)
        self.kx = np.where(i < nx // 2, i * (1.0 / self.lx), i * (1.0 / self.lx) - nx / self.lx)
        self.ky = np.where(j < ny // 2, j * (1.0 / self.ly), j * (1.0 / self.ly) - ny / self.ly)
        self.k2 = self.kx[:, None] * self.kx[:, None] + self.ky[None, :] * self.ky[None, :]
        self.bw_potential = min(nx / (2 * self.lx), ny / (2 * self.ly))
        self.bw = (2.0 / 3.0) * self.bw_potential
        self.s = math.sqrt(nx * ny)
        self.keep = self.put(self.k2 < self.bw ** 2)

    def put(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), device=self.dev)

    def back(self, a):
        return torch.fft.ifft2(a, norm="forward")

    def propagator(self, thick):
        p = [np.where(np.abs(k) < self.bw, np.exp(-1j * _PI * self.lam * thick * k ** 2), 0.0)
             for k in (self.kx, self.ky)]
        return self.put(p[0])[:, None] * self.put(p[1])[None, :]

    def transmission(self, q, z):
        """Band-limited e^{i sigma V} of one slice."""
        v = torch.zeros((self.nx, self.ny), dtype=torch.complex128, device=self.dev)
        for zz in np.unique(z):
            h = np.zeros((self.nx, self.ny))
            at = q[z == zz]
            np.add.at(h, ([_snap(self.x, a, 0) for a in at[:, 0]],
                          [_snap(self.y, a, 0) for a in at[:, 1]]), 1.0)
            p, k2 = _KIRKLAND[int(zz)], self.k2
            f = (p[0] / (k2 + p[3]) + p[1] / (k2 + p[4]) + p[2] / (k2 + p[5]) +
                 p[6] * np.exp(-p[9] * k2) + p[7] * np.exp(-p[10] * k2) +
                 p[8] * np.exp(-p[11] * k2))
            f = np.where(k2 < self.bw_potential ** 2, f, 0.0)
            f = f * (self.lam * self.gam / (self.lx * self.ly))
            v += torch.fft.fft2(self.put(h).to(torch.complex128)) * self.put(f)
        v = self.back(v) / self.s
        t = torch.exp(-v.imag) * torch.exp(1j * v.real)
        return self.back(torch.fft.fft2(t) * self.keep) / (self.nx * self.ny)

    def probe(self, optics):
        corrected, cs3, cs5, defocus, alpha = optics
        lsq = self.lam * self.lam
        kl = self.k2 * lsq
        chi = _PI * self.lam * self.k2 * (0.5 * cs3 * kl - defocus +
                                          ((1.0 / 3.0) * cs5 * kl * kl if corrected else 0.0))
        p = self.back(self.put(np.where(kl < alpha * alpha, np.exp(-1j * chi), 0.0)))
        return p / torch.sqrt((p.abs() ** 2).sum())

    def shifts(self, case):
        xp, yp = _raster_points(case)
        out, sx, sy = [], 0, 0
        for a in xp:
            for b in yp:
                sx, sy = _snap(self.x, a, sx), _snap(self.y, b, sy)
                out.append((sx, sy))
        return out

    def mtf(self):
        """The detector MTF in k-space, band-limited as the program does."""
        x, y = self.lx ** 2 * self.kx / self.nx, self.ly ** 2 * self.ky / self.ny
        r = np.sqrt(x[:, None] ** 2 + y[None, :] ** 2)
        d = 0.5 * MTF_RATE * np.array(MTF_DOMAIN)
        v = np.where(r ** 2 < d[-1] ** 2, np.interp(r, d, MTF_VALUE), 0.0)
        v = v * np.sinc(x / MTF_RATE / np.pi)[:, None] * np.sinc(y / MTF_RATE / np.pi)[None, :]
        a = self.back(self.put(v).to(torch.complex128)) * self.keep
        return torch.fft.fft2(a) / (self.nx * self.ny)

    def detected(self, psi, mtf, alpha):
        """|psi| without the direct beam through the detector MTF."""
        far = self.put(self.lam ** 2 * self.k2 > alpha * alpha)
        w = self.back((psi.abs() * far).to(torch.complex128))
        re = (w.real * mtf.real - w.imag * mtf.imag) / self.s
        im = (re * mtf.imag + w.imag * mtf.real) / self.s
        return torch.fft.fft2(torch.complex(re, im)) / self.s * self.keep


def _exact_raster(case, configurations):
    """One simulation's results; several configurations are averaged."""
    cell = _Cell(case)
    optics, keep = _optics(case), (np.float32 if case["precision"] == "fp32" else np.float64)
    probe, shifts = cell.probe(optics), cell.shifts(case)
    stacks = []
    for q, z in configurations:
        lists, thick = _slices(q)
        stacks.append([(cell.transmission(q[a], z[a]), cell.propagator(d))
                       for a, d in zip(lists, thick)])
    modes = _modes(case)
    # rings 0 < k <= (n + 1) dk; the last segment collects what lies outside
    dk = 1.2065 * math.sqrt(cell.kx[1] ** 2 + cell.ky[1] ** 2)
    nk = int(cell.bw / dk)
    bounds = np.arange(nk + 1) * dk
    bins = np.searchsorted(bounds[1:] * bounds[1:], cell.k2.reshape(-1), "left")
    counts = np.bincount(bins, minlength=nk + 1)[:nk].astype(np.int32)
    inside = cell.lam * bounds[1:] <= optics[4]
    ring = cell.put(bins)

    def ring_sum(a):
        out = torch.zeros(nk + 1, dtype=torch.float64, device=cell.dev)
        return out.index_add_(0, ring, a.reshape(-1)).cpu().numpy()[:nk]

    annulus = cell.put((cell.k2 > DET_INNER / cell.lam) & (cell.k2 <= DET_OUTER / cell.lam))
    mtf = cell.mtf() if case["mtf"] else None
    adf, amp, inten = [], [], []
    acc_a = torch.zeros((cell.nx, cell.ny), dtype=torch.float64, device=cell.dev)
    acc_i = torch.zeros_like(acc_a)
    for sx, sy in shifts:
        wave, signal = 0.0, 0.0
        for stack in stacks:
            psi = torch.fft.fft2(torch.roll(probe, (sx, sy), (0, 1))) / cell.s
            for t, p in stack:
                psi = cell.back(psi)
                re = (t.real * psi.real - t.imag * psi.imag) / cell.s
                im = (t.real * psi.imag + t.imag * re) / cell.s
                psi = torch.fft.fft2(torch.complex(re, im)) / cell.s * cell.keep * p
            signal = signal + (psi.abs() ** 2 * annulus).sum() / len(stacks)
            wave = wave + psi / len(stacks)
        adf.append(signal)
        if modes:
            wave = cell.detected(wave, mtf, optics[4]) if case["mtf"] else wave
            a = wave.abs()
            amp.append(ring_sum(a))
            inten.append(ring_sum(a * a))
            acc_a += a
            acc_i += a * a
    out = {"adf_image": torch.stack(adf).cpu().numpy().reshape(case["rx"], case["ry"]).astype(keep),
           "bin_counts": counts if modes else np.zeros(0, np.int32)}
    if case["waves"]:
        out["final_psi"] = torch.view_as_real(wave).cpu().numpy().astype(keep)
    n, c = len(shifts), counts.astype(np.float64)
    with np.errstate(all="ignore"):
        s1 = np.where(inside, 0.0, np.array(amp).reshape(-1, nk) if modes else 0.0)
        s2 = np.where(inside, 0.0, np.array(inten).reshape(-1, nk) if modes else 0.0)
        m_a, m_i = acc_a / n, acc_i / n
        r_i, r_q, r_a = (np.where(inside, 0.0, ring_sum(a)) for a in (m_i, m_a * m_a, m_a))
        direct = cell.put(cell.lam ** 2 * cell.k2 <= optics[4] ** 2)
        r_v = np.where(inside, 0.0, ring_sum(torch.where(direct, 0.0, m_i / (m_a * m_a) - 1.0)))
        total = (s1 / c).sum(0)
        v = {"V_omega": np.where(total == 0.0, 0.0,
                                 n * ((s1 / c) ** 2).sum(0) / (total * total) - 1.0),
             "Vbar_r": ((s2 / c) / (s1 / c) ** 2 - 1.0).sum(0) / n,
             "V_gt17": (r_i / c) / (r_q / c), "V_re": (r_i / c) / (r_a / c) ** 2 - 1.0,
             "V_rbar": (r_q / c) / (r_a / c) ** 2 - 1.0, "Omega_vimage": r_v / c}
    out.update({m: v[m].astype(keep) for m in modes})
    return out


def exact(case, seed):
    outs = []
    for k, c in enumerate(_rasters(case)):
        outs.append(_exact_raster(c, _snapshot_atoms(c, 1000 * seed + k)))
    return outs[0] if case["kind"] in ("run", "build", "md") else outs
