"""Rounding of the slice passes: the exit wave's error against a long-double
restatement of its slices, beside the error of the passes' own arithmetic restated
on the host.

The restatement transforms with the passes' radices: one twiddle product a stage,
then a radix-R butterfly by decimation in frequency, 32 points as 4 x 8 and 16 as
4 x 4, a product's second half contracted.  Lengths that do just that have to
round as it does: 5 % for the order of the scale factors and for the sampling of
the rms (0.4 % from 2e4 values).  Lengths whose later stages fuse their products
into the layers round by up to 1.14 of it in a single transform (random and
decaying input, forward and inverse, in emulated FP32): 15 %.  The error is taken
outside the aperture, where the wave is all scattered."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu

PI = 3.14159265369  # the program's constant
ALPHA = 0.010
RADICES = {64: (8, 8), 128: (16, 8), 256: (16, 16), 512: (32, 16), 1024: (32, 32),
           2048: (32, 8, 8), 4096: (32, 32, 4)}
ROW64_RADICES = {**RADICES, 2048: (16, 16, 8), 4096: (16, 16, 16)}
ROW32_RADICES = {**RADICES, 4096: (16, 16, 16)}


class _Arithmetic:
    """Transforms along axis 0 of (real, imaginary) pairs in one precision."""

    def __init__(self, real):
        self.real = real
        self.wide = np.float64 if real is np.float32 else np.longdouble

    def fma(self, a, b, c):
        return (a.astype(self.wide) * b + c).astype(self.real)

    def turn(self, a, num, den):
        """a W_den^num; num a number or one per element of the second axis."""
        if np.ndim(num) == 0 and 4 * num % den == 0:
            q = 4 * num // den % 4
            return (a, (a[1], -a[0]), (-a[0], -a[1]), (-a[1], a[0]))[q]
        x = 2 * np.arccos(np.longdouble(-1)) * np.asarray(num, np.longdouble) / den
        c, s = np.cos(x).astype(self.real), (-np.sin(x)).astype(self.real)
        return self.fma(a[0], c, -(a[1] * s)), self.fma(a[0], s, a[1] * c)

    def dif(self, u):
        n = len(u)
        if n == 1:
            return u
        low = [(x[0] + y[0], x[1] + y[1]) for x, y in zip(u, u[n // 2:])]
        high = [self.turn((x[0] - y[0], x[1] - y[1]), k, n)
                for k, (x, y) in enumerate(zip(u, u[n // 2:]))]
        out = [None] * n
        out[0::2], out[1::2] = self.dif(low), self.dif(high)
        return out

    def butterfly(self, u):
        n = len(u)
        if n < 16:
            return self.dif(u)
        m = n // 4
        first = [self.dif(u[k::m]) for k in range(m)]  # [n2][k1]
        out = [None] * n
        for k1 in range(4):
            out[k1::4] = self.dif([self.turn(first[n2][k1], n2 * k1, n) for n2 in range(m)])
        return out

    def forward(self, a, radices):
        """a: complex, transformed along axis 0."""
        n = a.shape[0]
        v, done = (a.real.astype(self.real), a.imag.astype(self.real)), 1
        for radix in radices:
            j = np.arange(n // radix)
            k = (j % done)[:, None]
            u = [(v[0][j + r * len(j)], v[1][j + r * len(j)]) for r in range(radix)]
            if done > 1:
                u = [u[0]] + [self.turn(u[r], r * k, done * radix) for r in range(1, radix)]
            y = self.butterfly(u)
            at = (j // done) * done * radix + j % done
            v = np.empty_like(v[0]), np.empty_like(v[1])
            for r in range(radix):
                v[0][at + r * done], v[1][at + r * done] = y[r]
            done *= radix
        return v[0] + v[1] * np.array(1j, np.result_type(self.real, np.complex64))

    def fft2(self, a, rows, cols):
        return self.forward(self.forward(a.T, rows[a.shape[1]]).T, cols[a.shape[0]])

    def ifft2(self, a, rows, cols):
        return self.forward(self.forward(a.conj(), cols[a.shape[0]]).T, rows[a.shape[1]]).T.conj()


class _Steps:
    """The slices of a specimen restated in numpy (transforms without factors)."""

    def __init__(self, nx, ny, box, spec, probe):
        lam = msf.wavelength(200000.0)[0]
        kx, ky = np.fft.fftfreq(nx, box[0] / nx), np.fft.fftfreq(ny, box[1] / ny)
        k2 = kx[:, None] ** 2 + ky[None, :] ** 2
        bw = (2.0 / 3.0) * min(nx / (2 * box[0]), ny / (2 * box[1]))
        self.keep = k2 < bw ** 2
        self.outside = self.keep & (k2 * lam * lam > (1.01 * ALPHA) ** 2)
        s = spec.slices()
        self.t = [_complex(spec.transmission(k)) for k in range(s["n"])]
        self.prop = [(np.exp(-1j * PI * lam * d * kx ** 2), np.exp(-1j * PI * lam * d * ky ** 2))
                     for d in s["thickness"]]
        self.probe, self.s = probe, np.sqrt(nx * ny)

    def _leave(self, psi, px, py):
        """Band limit and propagator, in psi's precision."""
        px, py = px.astype(psi.dtype), py.astype(psi.dtype)
        return psi * self.keep * (px[:, None] * py[None, :])

    def whole(self, c, fft2, ifft2):
        """The wave itself, every step in precision c."""
        s = np.sqrt(c(self.keep.size)).real
        psi = fft2(self.probe.astype(c)) / s
        for t, (px, py) in zip(self.t, self.prop):
            psi, t = ifft2(psi), t.astype(c)
            re = (t.real * psi.real - t.imag * psi.imag) / s
            im = (t.real * psi.imag + t.imag * re) / s
            psi = self._leave(fft2(re + c(1j) * im) / s, px, py)
        assert psi.dtype == c
        return psi

    def scattered(self, fft2, ifft2):
        """Its scattered part in FP32, on top of the FP64 vacuum wave."""
        c, i = np.complex64, np.float32(1.0 / self.s)
        vac, d = np.fft.fft2(self.probe) / self.s, np.zeros(self.keep.shape, c)
        for t, (px, py) in zip(self.t, self.prop):
            p = np.fft.ifft2(vac, norm="forward")
            vac = self._leave(np.fft.fft2(p) / self.s ** 2, px, py)
            tau, p, d = (t - 1.0).astype(c), p.astype(c), ifft2(d)
            re = (tau.real * p.real - tau.imag * p.imag + d.real + tau.real * d.real -
                  tau.imag * d.imag) * i
            im = (tau.real * p.imag + d.imag + tau.real * d.imag +
                  tau.imag * (p.real * i + re)) * i
            d = self._leave(fft2(re + c(1j) * im) * i, px, py)
        assert d.dtype == c
        return vac + d


def _complex(a):
    return a[..., 0] + 1j * a[..., 1]


# every length of the column passes in its turn, and of the FP64 row pass
@pytest.mark.parametrize("precision,nx,ny,bound", [
    ("fp64", 64, 64, 1.05), ("fp64", 128, 128, 1.05), ("fp64", 256, 256, 1.05),
    ("fp64", 512, 64, 1.15), ("fp64", 64, 512, 1.15), ("fp64", 1024, 64, 1.15),
    ("fp64", 64, 1024, 1.15), ("fp64", 2048, 64, 1.15), ("fp64", 64, 2048, 1.15),
    ("fp64", 4096, 64, 1.15), ("fp64", 64, 4096, 1.15),
    ("fp32", 64, 64, 1.05), ("fp32", 128, 128, 1.05), ("fp32", 256, 256, 1.05),
    ("fp32", 512, 64, 1.05), ("fp32", 1024, 64, 1.15), ("fp32", 2048, 64, 1.05),
    ("fp32", 4096, 64, 1.05)])
def test_exit_wave_rounds_like_its_arithmetic(precision, nx, ny, bound):
    fp64 = precision == "fp64"
    host = _Arithmetic(np.float64 if fp64 else np.float32)
    radices = (ROW64_RADICES if fp64 else ROW32_RADICES), RADICES
    transforms = lambda a: host.fft2(a, *radices), lambda a: host.ifft2(a, *radices)
    box = np.array([nx * 0.1, ny * 0.1, 16.0])
    grid = msf.Grid(nx=nx, ny=ny, voltage=200000.0, xperiod=box[0], yperiod=box[1],
                    zperiod=box[2], dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0,
                    ymin=0.0, zmin=0.0, min_slice=2.0)
    zero = np.zeros(1)
    raster = msf.Raster(1, 1, zero.ctypes.data_as(msf._dp), zero.ctypes.data_as(msf._dp))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=ALPHA)
    det = msf.Detect(outputs=msf.OUT_ADF_IMAGE, det_inner=0.04, det_outer=0.2, dr=1.0)
    ours = theirs = 0.0
    for seed in range(max(1, 65536 // (nx * ny))):
        q = np.random.default_rng(seed).uniform(0.0, 1.0, (max(20, int(0.03 * box.prod())), 3))
        z = np.full(len(q), 14, np.uint32)
        ctx, ctx64 = msf.Context(precision=precision), msf.Context(precision="fp64")
        got = _complex(ctx.run(ctx.specimen(grid, q * box, z), optics, raster, det,
                               want_final_psi=True).final_psi_2d)
        spec = ctx64.specimen(grid, q * box, z)
        steps = _Steps(nx, ny, box, spec, _complex(ctx64.probe(spec, optics)))
        exact = steps.whole(np.clongdouble, np.fft.fft2,
                            lambda a: np.fft.ifft2(a, norm="forward"))
        same = steps.whole(np.complex128, *transforms) if fp64 else steps.scattered(*transforms)
        m = steps.outside
        ours += float((np.abs(got - exact)[m] ** 2).sum())
        theirs += float((np.abs(same - exact)[m] ** 2).sum())
    assert ours <= bound ** 2 * theirs, np.sqrt(ours / theirs)
