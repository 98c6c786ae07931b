"""
Reconstructions whose time this repository tracks: whole calls of the public classes, from the constructor to
both read-outs, over the algorithms, mesh sizes, precisions, lines of sight and catalogues the package is used
for.  ``run`` is what a user's program does for one reconstruction; ``exact`` is the same reconstruction in plain
torch, 64 bits throughout.
"""
import math

import numpy as np
import torch

import pyrecon_b200
from pyrecon_b200 import mocks

CLASSES = {'iterative': 'IterativeFFTReconstruction', 'plane_parallel': 'PlaneParallelFFTReconstruction',
           'multigrid': 'MultiGridReconstruction', 'original_multigrid': 'OriginalMultiGridReconstruction',
           'particle': 'IterativeFFTParticleReconstruction'}
F, BIAS, RADIUS = 0.8, 2.0, 15.0


def case(name, algorithm, nmesh, cell, ndata, nrandoms, los='local', dtype='f4', pos='f4', weighted=False, wrap=False,
         host=False, real_smoothing=False):
    """One reconstruction: mesh of ``nmesh`` cells of about ``cell`` Mpc/h (box lengths are whole numbers), a
    catalogue of ``ndata`` lognormal points and ``nrandoms`` uniform randoms (0: a periodic box without randoms)."""
    nx, ny, nz = (nmesh,) * 3 if isinstance(nmesh, int) else nmesh
    c = dict(algorithm=algorithm, nx=nx, ny=ny, nz=nz, lx=max(1, round(nx * cell)), ly=max(1, round(ny * cell)),
             lz=max(1, round(nz * cell)), ndata=ndata, nrandoms=nrandoms, los=los, dtype=dtype, pos=pos,
             weighted=weighted, wrap=wrap, host=host, real_smoothing=real_smoothing)
    if name:
        c['name'] = name
    return c


def listed():
    return [
        # the headline workload: a survey volume at the full mesh size, local line of sight
        case('iterative_512', 'iterative', 512, 2000 / 512, 5_000_000, 20_000_000),
        # a survey catalogue run in double precision (the package's default precision) with weights, 3 2^k mesh
        case('iterative_192_f8', 'iterative', 192, 10.0, 600_000, 2_400_000, dtype='f8', pos='f8', weighted=True),
        # a box whose sides are not alike: mesh from a cell size, so no powers of two, one odd axis
        case('iterative_ragged', 'iterative', (150, 125, 243), 8.0, 400_000, 1_600_000, los='x'),
        # numpy catalogues in, numpy positions out, as the reference's users hold them
        case('plane_parallel_256_host', 'plane_parallel', 256, 7.8125, 500_000, 2_000_000, los='z', pos='f8', host=True),
        # one of many periodic-box mocks
        case('plane_parallel_mock_128', 'plane_parallel', 128, 7.8125, 300_000, 0, los='z', wrap=True),
        # the smallest calls: a quick look at a small sample, default precision
        case('plane_parallel_64_f8', 'plane_parallel', 64, 15.625, 20_000, 80_000, los='z', dtype='f8', pos='f8'),
        # multigrid with weights, local line of sight, FP32 meshes and FP64 positions
        case('multigrid_256', 'multigrid', 256, 7.8125, 2_000_000, 10_000_000, pos='f8', weighted=True),
        # the largest: multigrid on the headline mesh
        case('multigrid_512', 'multigrid', 512, 2000 / 512, 5_000_000, 20_000_000),
        # periodic-box mock through multigrid, line of sight along an axis
        case('multigrid_mock_192', 'multigrid', 192, 1000 / 192, 1_000_000, 0, los='z', wrap=True),
        # a small multigrid run in double precision, where launches count
        case('multigrid_64_f8', 'multigrid', 64, 20.0, 50_000, 200_000, dtype='f8', pos='f8'),
        # iterations that repaint the particles, 3 2^k mesh
        case('particle_384', 'particle', 384, 2000 / 384, 2_000_000, 8_000_000),
        # Martin White's contrast and the truncated real-space smoothing
        case('original_multigrid_real_128', 'original_multigrid', 128, 7.8125, 1_000_000, 5_000_000, weighted=True,
             pos='f8', real_smoothing=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    algorithm = rng.choice(['iterative', 'iterative', 'plane_parallel', 'plane_parallel', 'multigrid', 'multigrid',
                            'particle', 'original_multigrid'])
    dtype = rng.choice(['f4', 'f4', 'f8'])
    top = {'iterative': 512, 'plane_parallel': 512, 'multigrid': 448, 'particle': 384,
           'original_multigrid': 192}[algorithm]
    if dtype == 'f8':
        top = min(top, 256)
    if 'multigrid' in algorithm:
        # the sizes the reference recommends: 2^k times 1, 3, 5 or 7
        nmesh = rng.choice([n for n in (48, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448) if n <= top])
    elif rng.random() < 0.4:
        nmesh = tuple(_log(rng, 40, min(top, 300)) for _ in range(3))    # from a cell size: any whole number
    else:
        nmesh = rng.choice([n for n in (48, 64, 96, 100, 128, 150, 192, 200, 256, 300, 384, 400, 512) if n <= top])
    cells = nmesh ** 3 if isinstance(nmesh, int) else nmesh[0] * nmesh[1] * nmesh[2]
    cell = rng.uniform(4.0, 10.0)
    ndata = min(5_000_000, _log(rng, 20_000, max(40_000, min(5_000_000, cells // 8))))
    periodic = algorithm != 'particle' and rng.random() < 0.4
    los = rng.choice(['x', 'y', 'z', 'diagonal'] + (['local', 'local', 'local'] if algorithm != 'plane_parallel' and
                                                    not periodic else []))
    # four randoms per data point, and enough of them for every smoothed cell to lie far above the threshold
    nrandoms = 0 if periodic else max(4 * ndata, min(20_000_000, cells // 4))
    if algorithm == 'original_multigrid':
        nrandoms = 0 if periodic else min(20_000_000, 2 * cells)
    return case(None, algorithm, nmesh, cell, ndata, nrandoms, los=los, dtype=dtype,
                pos=rng.choice(['f4', 'f8']) if dtype == 'f4' else 'f8', weighted=rng.random() < 0.3, wrap=periodic,
                host=False, real_smoothing=algorithm == 'original_multigrid' and rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------
# the user's program
# ---------------------------------------------------------------------------------------------

def _shape(c):
    return c['nx'], c['ny'], c['nz']


def _box(c):
    return np.array([c['lx'], c['ly'], c['lz']], dtype='f8')


def _centre(c):
    """Surveys sit away from the observer at the origin; periodic boxes start there."""
    return _box(c) / 2. if c['wrap'] else np.array([2000., 1500., 1800.])


def _los(c):
    return {'local': None, 'diagonal': [1., 1., 0.5]}.get(c['los'], c['los'])


def _catalogues(c, seed):
    """(data, data weights, randoms, random weights) on the device."""
    grid, low, box = 128, _centre(c) - _box(c) / 2., _box(c)
    tdtype = torch.float32 if c['pos'] == 'f4' else torch.float64

    # surveys keep a margin to the box's faces; a coordinate within rounding of the upper face, where an FP32
    # index rounds up to the mesh size, is left out of periodic boxes too
    margin = 0. if c['wrap'] else 1e-3

    def place(unit):
        unit = margin + unit * (1. - 2. * margin) * (1. - 2. ** -20)
        pos = torch.as_tensor(low, device='cuda') + unit * torch.as_tensor(box, device='cuda')
        return pos.to(tdtype).contiguous()

    data = place(mocks.lognormal_positions_torch(c['ndata'], grid, 1000., 500., seed=seed * 8 + 1,
                                                 field_seed=seed * 8 + 2) / 1000.)
    randoms = wd = wr = None
    if c['nrandoms']:
        randoms = place(mocks.uniform_positions_torch(c['nrandoms'], 1000., 500., seed=seed * 8 + 3) / 1000.)
    if c['weighted']:
        wd = mocks.weights_torch(c['ndata'], seed=seed * 8 + 4, dtype=c['pos'])
        if c['nrandoms']:
            wr = mocks.weights_torch(c['nrandoms'], seed=seed * 8 + 5, dtype=c['pos'])
    return data, wd, randoms, wr


def prepare(c, seed):
    cat = _catalogues(c, seed)
    if c['host']:
        cat = [None if t is None else t.cpu().numpy() for t in cat]
    return c, cat


def run(state):
    c, (data, wd, randoms, wr) = state
    cls = getattr(pyrecon_b200, CLASSES[c['algorithm']])
    recon = cls(f=F, bias=BIAS, los=_los(c), nmesh=_shape(c), boxsize=_box(c), boxcenter=_centre(c), dtype=c['dtype'],
                wrap=c['wrap'])
    recon.assign_data(data, wd)
    if randoms is not None:
        recon.assign_randoms(randoms, wr)
    if c['real_smoothing']:
        recon.set_density_contrast(smoothing_radius=RADIUS, method='real')
    else:
        recon.set_density_contrast(smoothing_radius=RADIUS)
    recon.run()
    if c['wrap']:
        # a periodic box: the displacements (a shifted position may fall on either side of a face)
        return {'data': recon.read_shifts(data)}
    out = {'data': recon.read_shifted_positions('data' if c['algorithm'] == 'particle' else data)}
    if randoms is not None:
        out['randoms'] = recon.read_shifted_positions(randoms, field='disp')
    return out


def work(c):
    """Catalogues read once and their results written once; the transforms of the smoothing and of the algorithm
    (5 N log2 N / 2 each for real data), or the multigrid schedule's sweeps; the particles' cloud-in-cell steps."""
    cells = c['nx'] * c['ny'] * c['nz']
    item = 4 if c['pos'] == 'f4' else 8
    particles = c['ndata'] + c['nrandoms']
    nbytes = particles * (6 * item + (item if c['weighted'] else 0))
    fft = 2.5 * cells * math.log2(cells)
    smooth = (4 if c['nrandoms'] else 2)
    if c['algorithm'] == 'iterative':
        n = smooth + 3 * (1 + (6 if c['los'] == 'local' else 1)) + 4
    elif c['algorithm'] == 'plane_parallel':
        n = smooth + 4
    elif c['algorithm'] == 'particle':
        n = smooth + 2 * 2 + 3 * 4
    else:
        n = smooth if not c['real_smoothing'] else 0
    flops = n * fft + particles * 100
    if 'multigrid' in c['algorithm']:
        flops += cells * 6 * 11 * 60 * 8 / 7
    return {'bytes': nbytes, 'flops': flops}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------

def _col(a, axis):
    return torch.as_tensor(np.asarray(a, dtype='f8'), device='cuda').reshape([-1 if i == axis else 1 for i in range(3)])


class _Exact(object):

    def __init__(self, c):
        self.c, self.n = c, _shape(c)
        self.box, self.centre = _box(c), _centre(c)
        self.cell = self.box / np.array(self.n)
        los = _los(c)
        if los is None:
            self.los = None
        else:
            los = np.eye(3)['xyz'.index(los)] if isinstance(los, str) else np.array(los)
            self.los = los / np.sqrt((los ** 2).sum())
        self.k = [_col(2 * np.pi * np.fft.fftfreq(n, d=d), i) for i, (n, d) in enumerate(zip(self.n, self.cell))]
        self.beta = F / BIAS

    def t(self, a):
        return torch.as_tensor(np.asarray(a, dtype='f8'), device='cuda')

    def wrapped(self, pos):
        low = self.t(self.centre - self.box / 2.)
        return torch.remainder(pos - low, self.t(self.box)) + low

    def corners(self, pos):
        x = ((pos - self.t(self.centre)) / self.t(self.box) + 0.5) * self.t(self.n)
        base = x.floor()
        frac = x - base
        base = base.long()
        for e in range(8):
            d = [(e >> 2) & 1, (e >> 1) & 1, e & 1]
            ijk = [(base[:, a] + d[a]) % self.n[a] for a in range(3)]
            w = 1.
            for a in range(3):
                w = w * (frac[:, a] if d[a] else 1. - frac[:, a])
            yield (ijk[0] * self.n[1] + ijk[1]) * self.n[2] + ijk[2], w

    def chunks(self, pos):
        return [pos[i:i + 4_000_000].double() for i in range(0, len(pos), 4_000_000)]

    def paint(self, pos, weights, wrap):
        mesh = torch.zeros(int(np.prod(self.n)), dtype=torch.float64, device='cuda')
        ws = [None] * len(self.chunks(pos)) if weights is None else [w.reshape(-1) for w in self.chunks(weights)]
        for p, w in zip(self.chunks(pos), ws):
            for i, cw in self.corners(self.wrapped(p) if wrap else p):
                mesh.index_add_(0, i, cw if w is None else cw * w)
        return mesh.reshape(self.n)

    def read(self, meshes, pos, wrap=False):
        out = []
        for p in self.chunks(pos):
            acc = torch.zeros_like(p)
            for i, w in self.corners(self.wrapped(p) if wrap else p):
                for a in range(3):
                    acc[:, a] += meshes[a].reshape(-1)[i] * w
            out.append(acc)
        return torch.cat(out)

    def smooth(self, mesh):
        g = [torch.exp(-0.5 * (RADIUS * k) ** 2) for k in self.k]
        return torch.fft.ifftn(torch.fft.fftn(mesh) * g[0] * g[1] * g[2]).real

    def smooth_real(self, mesh):
        """Convolution with the Gaussian cut at 2.5 sigma (its taps' sum divided out)."""
        sig = RADIUS / self.cell
        rad = [int(2.5 * s + 1.) for s in sig]
        d = [torch.arange(-r, r + 1, device='cuda', dtype=torch.float64) for r in rad]
        r2 = sum(_col((x / s).cpu().numpy() ** 2, a) for a, (x, s) in enumerate(zip(d, sig)))
        taps = torch.where(r2 < 2.5 ** 2, torch.exp(-r2 / 2), torch.zeros_like(r2))
        kernel = torch.zeros(self.n, dtype=torch.float64, device='cuda')
        idx = [(x.long() % n) for x, n in zip(d, self.n)]
        flat = (idx[0][:, None, None] * self.n[1] + idx[1][None, :, None]) * self.n[2] + idx[2][None, None, :]
        kernel.reshape(-1).index_add_(0, flat.reshape(-1), taps.reshape(-1))
        return torch.fft.ifftn(torch.fft.fftn(mesh) * torch.fft.fftn(kernel)).real / taps.sum()

    def contrast(self, data, randoms, nrandoms, ran_min=0.01):
        if randoms is None:
            return (data / data.mean() - 1.) / BIAS
        alpha = data.sum() / randoms.sum()
        mask = randoms > ran_min * randoms.sum() / nrandoms
        return torch.where(mask, (data - alpha * randoms) / (BIAS * alpha * randoms), torch.zeros_like(data))

    def contrast_original(self, data, randoms, ran_min=0.75):
        smooth = self.smooth_real if self.c['real_smoothing'] else self.smooth
        if randoms is None:
            return smooth((data / data.mean() - 1.) / BIAS)
        mask = randoms >= ran_min
        data = torch.where((randoms > 0) & ~mask, torch.zeros_like(data), data)
        alpha = data.sum() / randoms[mask].sum()
        delta = torch.where(mask, (data / (alpha * randoms) - 1.) / BIAS, torch.zeros_like(data))
        nonzero = delta != 0.
        return smooth(torch.where(nonzero, delta - delta[nonzero].mean(), delta))

    def inverse_laplacian(self, delta):
        dk = torch.fft.fftn(delta)
        k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        k2[0, 0, 0] = 1.
        dk /= k2
        dk[0, 0, 0] = 0.
        return dk, k2

    def psi(self, dk):
        return [torch.fft.ifftn(1j * self.k[a] * dk).real for a in range(3)]

    def iterative(self, delta, niterations=3):
        real = delta
        for it in range(niterations):
            dk, _ = self.inverse_laplacian(real)
            real = delta.clone()
            damp = self.beta / (1. + self.beta) if it == 0 else self.beta
            if self.los is not None:
                kl = sum(k * float(l) for k, l in zip(self.k, self.los))
                real -= damp * torch.fft.ifftn(kl ** 2 * dk).real
                continue
            x = [_col(self.centre[a] - self.box[a] / 2. + self.cell[a] * np.arange(self.n[a]), a) for a in range(3)]
            x2 = x[0] ** 2 + x[1] ** 2 + x[2] ** 2
            for i in range(3):
                for j in range(i, 3):
                    real -= (1. + (i != j)) * damp * x[i] * x[j] * torch.fft.ifftn(self.k[i] * self.k[j] * dk).real / x2
        return self.psi(self.inverse_laplacian(real)[0])

    def plane_parallel(self, delta):
        dk, k2 = self.inverse_laplacian(delta)
        mu2 = sum(k * float(l) for k, l in zip(self.k, self.los)) ** 2 / k2
        return self.psi(dk / (1. + self.beta * mu2))

    # -- multigrid: the reference's fixed full-multigrid schedule of damped-Jacobi V-cycles --

    def level(self, n):
        h = self.box / np.array(n)
        if self.los is None:
            p = [_col(np.arange(n[a]) + (self.centre[a] - self.box[a] / 2.) / h[a], a) for a in range(3)]
        else:
            p = [_col([self.los[a] / h[a]], a) for a in range(3)]
        g = self.beta / sum(h[a] ** 2 * p[a] ** 2 for a in range(3))
        return h, p, g

    def stencil(self, lev, v):
        h, p, g = lev
        roll = lambda u, a, s: torch.roll(u, -s, a)
        face = torch.zeros_like(v)
        rest = torch.zeros_like(v)
        for a in range(3):
            up, dn = roll(v, a, 1), roll(v, a, -1)
            s = up + dn
            face += s / h[a] ** 2
            s *= p[a] ** 2
            rest += s
            if self.los is None:
                rest += p[a] * (up - dn)
            d = up - dn
            for b in range(a + 1, 3):
                rest += 0.5 * p[a] * p[b] * (roll(d, b, 1) - roll(d, b, -1))
        face += g * rest
        diag = 2. * (sum(1. / h[a] ** 2 for a in range(3)) + g * sum(p[a] ** 2 for a in range(3)))
        return face, diag

    def jacobi(self, lev, v, f, niter=5, w=0.4):
        for _ in range(niter):
            s, diag = self.stencil(lev, v)
            s += f
            s /= diag
            v = (1. - w) * v + w * s
        return v

    @staticmethod
    def can_coarsen(n):
        return all(x > 4 and x % 2 == 0 for x in n)

    @staticmethod
    def reduce(r):
        for a in range(3):
            r = (2. * r + torch.roll(r, 1, a) + torch.roll(r, -1, a)) / 4.
            r = r.index_select(a, torch.arange(0, r.shape[a], 2, device='cuda'))
        return r

    @staticmethod
    def prolong(v):
        for a in range(3):
            v = torch.stack([v, 0.5 * (v + torch.roll(v, -1, a))], dim=a + 1).flatten(a, a + 1)
        return v

    def vcycle(self, n, v, f):
        lev = self.level(n)
        v = self.jacobi(lev, v, f)
        if self.can_coarsen(n):
            s, diag = self.stencil(lev, v)
            nc = tuple(x // 2 for x in n)
            fc = self.reduce(f - diag * v + s)
            v = v + self.prolong(self.vcycle(nc, torch.zeros_like(fc), fc))
        return self.jacobi(lev, v, f)

    def fmg(self, n, f):
        if self.can_coarsen(n):
            v = self.prolong(self.fmg(tuple(x // 2 for x in n), self.reduce(f)))
        else:
            v = torch.zeros_like(f)
        for _ in range(6):
            v = self.vcycle(n, v, f)
        return v

    def gradient(self, phi):
        return [(torch.roll(phi, -1, a) - torch.roll(phi, 1, a)) / (2. * self.cell[a]) for a in range(3)]

    # -- shifts --

    def along(self, shifts, pos):
        los = pos / (pos ** 2).sum(-1, keepdim=True).sqrt() if self.los is None else self.t(self.los)
        return (shifts * los).sum(-1, keepdim=True) * los

    def particle(self, data, wd, randoms, nrandoms):
        """Iterations on the data positions; returns (psi, reconstructed data positions)."""
        data = data.double()
        rec, mesh = data.clone(), self.smooth(self.paint(data, wd, False))
        randoms = self.smooth(randoms)
        for it in range(3):
            if it:
                mesh = self.smooth(self.paint(rec, wd, True))
            psi = self.psi(self.inverse_laplacian(self.contrast(mesh, randoms, nrandoms))[0])
            shifts = self.read(psi, rec, wrap=True)
            if it == 0:
                shifts = shifts - self.beta / (1. + self.beta) * self.along(shifts, data)
            rec = data - F * self.along(shifts, data)
        return psi, rec


def exact(c, seed):
    if c['nx'] * c['ny'] * c['nz'] > 512 ** 3:
        return None
    data, wd, randoms, wr = _catalogues(c, seed)
    x = _Exact(c)
    if c['algorithm'] == 'particle':
        psi, rec = x.particle(data, wd, x.paint(randoms, wr, False), c['nrandoms'])
        out = {'data': data.double() - (x.read(psi, rec, wrap=True) + data.double() - rec),
               'randoms': randoms.double() - x.read(psi, randoms)}
    else:
        dmesh = x.paint(data, wd, c['wrap'])
        rmesh = None if randoms is None else x.paint(randoms, wr, c['wrap'])
        if c['algorithm'] == 'original_multigrid':
            delta = x.contrast_original(dmesh, rmesh)
        else:
            delta = x.contrast(x.smooth(dmesh), None if rmesh is None else x.smooth(rmesh), c['nrandoms'])
        del dmesh, rmesh
        if 'multigrid' in c['algorithm']:
            psi = x.gradient(x.fmg(x.n, delta))
        else:
            psi = getattr(x, c['algorithm'])(delta)
        shifts = x.read(psi, data, wrap=c['wrap'])
        shifts = shifts + F * x.along(shifts, x.wrapped(data.double()) if c['wrap'] else data.double())
        if c['wrap']:
            out = {'data': shifts}
        else:
            out = {'data': data.double() - shifts}
            if randoms is not None:
                out['randoms'] = randoms.double() - x.read(psi, randoms)
    if c['host']:
        out = {k: v.cpu().numpy() for k, v in out.items()}
    return out
