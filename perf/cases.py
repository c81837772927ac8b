"""The workloads whose speed is measured: what users of this package run.

``listed()`` names them, ``draw`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (photons, model, the
reconstructor or problem object), ``run`` is one pass through the public
entry points and ``exact`` the same values by plain FP64 torch.

Photons are those of ``rspi.synth`` (Gaussian-blob objects, a sphere
reference, lognormal fluence); detector sizes, state grids, frame and photon
counts are those of its configurations, or smaller.
"""
import os
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, 'refspi-maxlp_b200')):
    if _p not in sys.path:
        sys.path.insert(0, _p)

_F8 = torch.float64

# kinds of work:
#   iterate    EMC.run_iteration: E-step, argmax, MaxLP M-step, host copies
#   posterior  E-step with the posterior window, then the weighted merge
#   fp64       E-step in the plain FP64 form
#   dense      E-step over densely stored frames (tensor-core form)
#   phaser     MaxLPhaser._run_phaser: host model and per-frame values in, model out
#   nll        MaxLP pixel NLL, value and gradient by autograd
#   slicenll   likelihood through model slicing, value and gradient by autograd
#   refine     MaxLPhaser._improve_model: support, difference map, error reduction


def _case(name, kind, size, frames, photons, rot=0, shifts=0, span=0., dias=0, modes=1,
          uneven=False, start='near', precision='fp32'):
    """``shifts`` values of either shift in [-span, span], ``dias`` diameters
    in [6, 8]; ``photons`` per frame (the median when ``uneven``: lognormal
    counts in [50, 50000]); ``start``: a random model (a first iteration) or
    one near the object (a later one)."""
    return dict(name=name, kind=kind, size=size, frames=frames, photons=photons, rot=rot,
                shifts=shifts, span=span, dias=dias, modes=modes, uneven=uneven, start=start,
                precision=precision)


def listed():
    return [
        # a try-out of a few dozen frames on a small detector: launches and latency
        _case('iterate_tiny', 'iterate', 41, 60, 300., 12, 3, 1., 2, start='random'),
        # the plain small reconstruction, its first iteration
        _case('iterate_small', 'iterate', 101, 1000, 500., 180, 7, 3., 5, start='random'),
        # the production reconstruction, an iteration from a model near the object
        _case('iterate_production', 'iterate', 185, 20000, 2000., 180, 9, 4., 5),
        # a heterogeneous sample as three models, photon counts over three decades
        _case('iterate_uneven_modes', 'iterate', 185, 4001, 1581., 180, 5, 2., 3, modes=3,
              uneven=True),
        # posteriors of every state and the posterior-weighted intensities
        _case('posterior_merge', 'posterior', 185, 1003, 2000., 60, 5, 2., 3, start='random'),
        # the FP64 form, chosen where every likelihood is wanted in FP64
        _case('estep_fp64', 'fp64', 101, 500, 500., 90, 5, 2., 3),
        # high-fluence frames stored densely
        _case('estep_dense', 'dense', 255, 600, 2.e5, 360, 3, 1., 3),
        # the M-step on its own, with host arrays as the E-step's user holds them
        _case('phaser_small', 'phaser', 101, 1000, 500., 180, 7, 3., 5),
        # one step of a gradient-based update of a float32 model over the
        # production frames
        _case('nll_gradient', 'nll', 185, 20000, 2000.),
        # the same in FP64, as the comparison of model updates evaluates it
        _case('nll_gradient_fp64', 'nll', 101, 1000, 500., precision='fp64'),
        # one step of fitting model, diameters, shifts and scales through slicing
        _case('slice_nll_gradient', 'slicenll', 185, 5000, 2000.),
        # model refinement between reconstructions
        _case('refine', 'refine', 185, 20, 500.),
    ]


def draw(rng):
    kind = rng.choice(['iterate'] * 4 + ['posterior', 'fp64', 'dense', 'phaser', 'nll', 'nll',
                       'slicenll', 'refine'])

    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    start = rng.choice(['random', 'near'])
    if kind == 'iterate':
        size = rng.randint(41, 185)
        rot, shifts, dias = rng.randint(12, 180), rng.randint(2, 7), rng.randint(2, 5)
        modes = rng.choice([1, 1, 1, 2, 3])
        most = int(4e8 / (rot * shifts * shifts * dias * modes))
        return _case('', kind, size, max(60, min(log(60, 20000), most)), float(log(200, 2000)),
                     rot, shifts, 0.5 * (shifts - 1), dias, modes, rng.random() < 0.3, start)
    if kind == 'posterior':
        return _case('', kind, rng.randint(61, 185), log(50, 1500), float(log(200, 2000)),
                     rng.randint(20, 90), rng.randint(2, 5), 2., rng.randint(2, 3), start=start)
    if kind == 'fp64':
        return _case('', kind, rng.randint(41, 151), log(50, 1500), float(log(100, 1000)),
                     rng.randint(12, 90), rng.randint(2, 5), 2., rng.randint(2, 3), start=start)
    if kind == 'dense':
        return _case('', kind, rng.randint(101, 255), log(50, 600), float(log(50000, 200000)),
                     rng.randint(60, 360), rng.randint(2, 3), 1., rng.randint(2, 3))
    if kind == 'phaser':
        return _case('', kind, rng.randint(41, 151), log(60, 5000), float(log(200, 2000)),
                     rng.randint(24, 180), rng.randint(3, 9), 3., rng.randint(2, 5), start=start)
    if kind == 'nll':
        if rng.random() < 0.3:
            return _case('', kind, rng.randint(41, 121), log(100, 1500), float(log(200, 1000)),
                         precision='fp64')
        return _case('', kind, rng.randint(61, 185), log(200, 20000), float(log(200, 2000)))
    if kind == 'slicenll':
        return _case('', kind, rng.randint(61, 185), log(200, 8000), float(log(200, 2000)))
    return _case('', kind, rng.randint(61, 255), rng.randint(10, 40), 500., start=start)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _data(case, seed):
    """Photons (host lists in the photons-file layout) and a start model."""
    from rspi import synth
    kw = {}
    if case['modes'] > 1:
        kw.update(n_modes=case['modes'],
                  mode_weights=[w / case['modes'] for w in range(1, case['modes'] + 1)])
    if case['uneven']:
        kw.update(count_lognormal=(case['photons'], 1.15, 50., 50000.))
    if case['kind'] == 'dense':
        # a flat background, half of a 2e5-photon frame on a 255^2 detector
        kw.update(dense=True, bg_level=0.5 * case['photons'] / (0.785 * case['size'] ** 2))
    big = case['size'] >= 150
    data = synth.generate(case['size'], case['frames'], case['photons'], 40 if big else 20,
                          20. if big else min(12., case['size'] / 8.), 0.5 if big else 0.3,
                          (6., 8.), 3., seed=int(seed), device='cuda', **kw)
    rng = np.random.default_rng([int(seed), 1])
    shape = np.shape(data['fsample'])
    if case['start'] == 'random':
        model = rng.random(shape) + 1j * rng.random(shape)
    else:
        # the object's transform, in units of the reference amplitude, 10% off
        noise = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        model = data['fsample'] / float(data['rel_scale']) * (1. + 0.07 * noise)
    return data, np.ascontiguousarray(model, dtype=np.complex128)


def _grid(case):
    """``lo hi n`` of the shifts and of the diameters."""
    return (-case['span'], case['span'], case['shifts']), (6., 8., case['dias'])


def _states(case):
    from rspi import geometry
    sh, dia = _grid(case)
    return geometry.state_grid(sh, sh, dia)


def _nearest_states(case, data):
    """Each frame's (shift x, shift y, diameter, angle) on the state grid, the
    grid point nearest its true values: what an E-step hands to the phaser."""
    sh, dia = _grid(case)

    def near(v, g):
        axis = np.linspace(*g)
        return axis[np.abs(np.asarray(v)[:, None] - axis[None]).argmin(1)]

    # the data generator turns the detector, the phaser the model
    j = np.rint(np.asarray(data['true_angles']) / np.pi * case['rot']).astype(int) % case['rot']
    return (near(data['true_shifts'][:, 0], sh), near(data['true_shifts'][:, 1], sh),
            near(data['true_diameters'], dia), j * np.pi / case['rot'])


def _device_photons(case, data, scaling=True):
    from rspi.device import DevicePhotons
    return DevicePhotons(data['ones'], data['multi'], data['place_ones'], data['place_multi'],
                         data['count_multi'], case['size'] ** 2, scaling,
                         frames=data.get('frames'))


def _leaves(case, data, model):
    """The differentiable inputs, model parts and per-frame parameters: in
    float32 for a float32 model (the adjoint configuration), else float64."""
    dt = torch.float32 if case['precision'] == 'fp32' else _F8
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype='f8')).to('cuda', dt)  # noqa
    return [t(model.real), t(model.imag), t(data['true_diameters']),
            t(data['true_shifts'][:, 0]), t(data['true_shifts'][:, 1]), t(data['scale'])]


def _photon_file(folder, data):
    from rspi.photonfile import write_photons
    return write_photons(os.path.join(folder, 'photons.npz'), data)


def prepare(case, seed):
    data, model = _data(case, seed)
    kind, size = case['kind'], case['size']
    if kind == 'iterate':
        from emc import EMC
        with tempfile.TemporaryDirectory() as tmp:
            _photon_file(tmp, data)
            out = tempfile.mkdtemp()
            sh, dia = _grid(case)
            with open(os.path.join(tmp, 'config.ini'), 'w') as f:
                f.write('[emc]\nsize = %d\nin_photons_file = photons.npz\noutput_folder = %s/\n'
                        'log_file = %s/EMC.log\nneed_scaling = True\nnum_rot = %d\n'
                        'num_modes = %d\nshiftx = %s\nshifty = %s\nsphere_dia = %s\n'
                        % (size, out, out, case['rot'], case['modes'], '%g %g %d' % sh,
                           '%g %g %d' % sh, '%g %g %d' % dia))
            rec = EMC(os.path.join(tmp, 'config.ini'))
        return dict(kind=kind, rec=rec, model=model)
    if kind in ('posterior', 'fp64', 'dense'):
        from rspi import geometry
        from rspi.device import EStep, Merge
        ph = _device_photons(case, data)
        gx, gy, gd, _ = _states(case)
        bg = data.get('bg', np.zeros(size ** 2))
        form = 'screen' if kind == 'posterior' else kind
        es = EStep(ph, size, case['rot'], gx, gy, gd, geometry.emc_masks(size)[1], bg, form=form)
        state = dict(kind=kind, es=es, model=torch.from_numpy(model).cuda())
        if kind == 'posterior':
            state['merge'] = Merge(es)
        return state
    if kind in ('phaser', 'refine'):
        from maxLP import MaxLPhaser
        from dset import Dataset
        with tempfile.TemporaryDirectory() as tmp:
            ds = Dataset(_photon_file(tmp, data), size ** 2, True)
        ph = MaxLPhaser(None, size, dataset=ds)
        if kind == 'refine':
            return dict(kind=kind, phaser=ph, model=torch.from_numpy(model).cuda())
        return dict(kind=kind, phaser=ph, model=model, values=_nearest_states(case, data))
    if kind == 'nll':
        from rspi.adjoint import NLLProblem
        prob = NLLProblem(_device_photons(case, data), size, data['true_angles'],
                          precision=case['precision'])
        pixels = prob.pixels
        leaves = _leaves(case, data, model[pixels])
    else:
        from rspi import geometry
        from rspi.adjoint import EMCNLLProblem
        leaves = _leaves(case, data, model)
        cs = np.stack([np.cos(data['true_angles']), np.sin(data['true_angles'])], 1)
        mask = geometry.emc_masks(size)[1]
        prob = EMCNLLProblem(_device_photons(case, data), size, cs, mask, np.zeros(size ** 2),
                             _vscale(case, data, model, mask), precision=case['precision'])
    for v in leaves:
        v.requires_grad_(True)
    return dict(kind=kind, problem=prob, leaves=leaves)


def _vscale(case, data, model, mask):
    """Photons per unit of model intensity over the likelihood pixels."""
    n1, nm = len(data['place_ones']), data['count_multi'].astype('f8')
    sel = mask < 1
    total = float(sel[data['place_ones']].sum()) if n1 else 0.
    total += float(nm[sel[data['place_multi']]].sum())
    return total / data['scale'].sum() / float((2. * np.abs(model[sel]) ** 2).sum())


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state['kind']
    if kind == 'iterate':
        rec = state['rec']
        rec.model = state['model']
        rec.run_iteration()
        return dict(model=rec.model, rmax=rec.rmax)
    if kind in ('posterior', 'fp64', 'dense'):
        es = state['es']
        es.run(state['model'])
        maxll, rmax, logz = es.reduce()
        out = dict(maxll=maxll, rmax=rmax, logz=logz, prob=es.frame_prob())
        if kind == 'posterior':
            out['intens'] = state['merge'].run()
        return out
    if kind == 'phaser':
        return state['phaser']._run_phaser(state['model'], *state['values'])
    if kind == 'refine':
        return state['phaser']._improve_model(state['model'])
    from rspi import adjoint
    fn = adjoint.nll if kind == 'nll' else adjoint.emc_nll
    leaves = state['leaves']
    loss = fn(state['problem'], *leaves).to(leaves[0].dtype)   # the program's own type
    return dict(loss=loss.detach(), grads=torch.autograd.grad(loss, leaves))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Inputs once, outputs once; flops: two per (photon on a likelihood
    pixel, state) and the other stages' own arithmetic.  About an eighth of a
    frame's photons lie on likelihood pixels (all pixels' counts, dense)."""
    size, n = case['size'], case['frames']
    npix = size * size
    phot = n * (case['photons'] * (1.9 if case['uneven'] else 1.))
    sel = 0.72 * npix
    n0 = case['shifts'] ** 2 * case['dias'] * case['modes']
    rows = n0 * case['rot']
    lists = 4. * min(phot, n * npix) + 16. * n
    model = 16. * npix * case['modes']
    kind = case['kind']
    likelihood = 2. * rows * phot / 8. + 12. * rows * sel
    pattern = case['modes'] * 0.78 * npix * 1089. * 10. * 8. * max(1, min(n0, phot / npix * 2))
    if kind == 'iterate':
        return dict(bytes=lists + 2 * model + 4. * n, flops=likelihood + pattern)
    if kind == 'posterior':
        return dict(bytes=lists + model + 4. * rows * n + 8. * n0 * npix, flops=likelihood)
    if kind == 'fp64':
        return dict(bytes=lists + model + 8. * rows * n, flops=likelihood)
    if kind == 'dense':
        return dict(bytes=2. * n * npix + model + 4. * rows * n,
                    flops=2. * rows * n * sel + 12. * rows * sel)
    if kind == 'phaser':
        return dict(bytes=lists + 2 * model + 32. * n, flops=pattern)
    if kind in ('nll', 'slicenll'):
        return dict(bytes=lists + 2 * model + 64. * n, flops=40. * n * sel + 100. * phot)
    return dict(bytes=2 * model, flops=62. * 8. * npix * size)


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _counts(case, data, dtype=_F8):
    """Photon counts, frames x pixels."""
    n, npix = case['frames'], case['size'] ** 2
    dev = torch.device('cuda')
    out = torch.zeros(n * npix, dtype=dtype, device=dev)
    for rows, place, cnt in ((data['ones'], data['place_ones'], None),
                             (data['multi'], data['place_multi'], data['count_multi'])):
        d = torch.repeat_interleave(torch.arange(n, device=dev),
                                    torch.as_tensor(rows).to(dev).long())
        p = torch.as_tensor(place).to(dev).long()
        v = torch.ones(p.numel(), dtype=dtype, device=dev) if cnt is None \
            else torch.as_tensor(cnt).to(dev, dtype)
        out.index_add_(0, d * npix + p, v)
    return out.view(n, npix)


def _axes(size):
    x = torch.arange(size, dtype=_F8, device='cuda') - size // 2
    return x[:, None].expand(size, size).reshape(-1), x[None].expand(size, size).reshape(-1)


def _sphere(s):
    return (torch.sin(s) - s * torch.cos(s)) / (s * s * s)


def _likelihood_pixels(size):
    x, y = _axes(size)
    r = torch.sqrt(x * x + y * y)
    keep = (r < size // 2) & (r >= size // 8) & (r >= 4)
    return torch.nonzero(keep).view(-1)


def _holo(size, model, sx, sy, dia, bg):
    """|M + reference|^2 + bg of one state."""
    x, y = _axes(size)
    s = torch.sqrt(x * x + y * y) * np.pi * dia / size
    ff = _sphere(torch.where(s == 0., torch.full_like(s, 1.e-5), s))
    th = 2. * np.pi * (x * sx + y * sy) / size
    re, im = torch.cos(th) * ff + model.real, torch.sin(th) * ff + model.imag
    return re * re + im * im + bg


def _footprint(size, cs, sn, x, y):
    """Corner index, fractions and validity of the rotated positions."""
    cen = size // 2
    tx, ty = x * cs - y * sn + cen, x * sn + y * cs + cen
    ix, iy = torch.floor(tx), torch.floor(ty)
    ok = (ix >= 0) & (ix <= size - 2) & (iy >= 0) & (iy <= size - 2)
    zero = torch.zeros_like(ix)
    ix, iy = torch.where(ok, ix, zero), torch.where(ok, iy, zero)
    return (ix * size + iy).long(), tx - ix, ty - iy, ok


def _corners(fx, fy, size):
    return ((0, (1 - fx) * (1 - fy)), (size, fx * (1 - fy)), (1, (1 - fx) * fy),
            (size + 1, fx * fy))


def _rotation_angles(case):
    ang = np.arange(case['rot']) * np.pi / case['rot']
    t = lambda a: torch.as_tensor(a).cuda()[:, None]  # noqa: E731
    return t(np.cos(ang)), t(np.sin(ang))


class _ExactEStep:
    """Likelihood rows in FP64, one (mode, shift, diameter) state at a time."""

    def __init__(self, case, data, model):
        self.case, size = case, case['size']
        self.sel = _likelihood_pixels(size)
        self.k = _counts(case, data)
        tot = self.k.sum(1)
        self.scales = tot / tot.mean()
        self.bg = torch.as_tensor(data['bg']).cuda() if 'bg' in data \
            else torch.zeros(size * size, dtype=_F8, device='cuda')
        models = torch.as_tensor(model).cuda().view(case['modes'], -1)
        gx, gy, gd, _ = _states(case)
        self.values = list(zip(gx, gy, gd))
        self.params = [(m,) + v for m in models for v in self.values]
        powder = self.k.mean(0)
        self.msum = torch.stack([_holo(size, m, a, b, d, self.bg)[self.sel].sum()
                                 for m, a, b, d in self.params])
        vscale = powder[self.sel].sum() / self.msum.sum() * len(self.params)
        self.init = -(self.msum * vscale)
        self.ksel_t = self.k[:, self.sel].t().contiguous()
        x, y = _axes(size)
        cs, sn = _rotation_angles(case)
        self.foot = _footprint(size, cs, sn, x[self.sel][None], y[self.sel][None])

    def rows(self, i):
        m, a, b, d = self.params[i]
        size = self.case['size']
        w = _holo(size, m, a, b, d, self.bg)
        base, fx, fy, ok = self.foot
        v = sum(w[base + o] * wt for o, wt in _corners(fx, fy, size)) + self.bg[self.sel][None]
        bad = ~ok | (v < 1.e-20)
        v = torch.where(bad, torch.full_like(v, -1000.), torch.log(torch.where(bad, 1., v)))
        return v @ self.ksel_t + self.init[i] * self.scales[None]

    def reduce(self, keep):
        n, r = self.case['frames'], self.case['rot']
        best = torch.full((n,), -np.inf, dtype=_F8, device='cuda')
        arg = torch.zeros(n, dtype=torch.int64, device='cuda')
        logz, prob = best.clone(), []
        for i in range(len(self.params)):
            ll = self.rows(i)
            v, j = ll.max(0)
            better = v > best
            best, arg = torch.where(better, v, best), torch.where(better, i * r + j, arg)
            logz = torch.logaddexp(logz, torch.logsumexp(ll, 0))
            if keep:
                prob.append(ll)
        return best, arg, logz, (torch.cat(prob) if keep else None)


def _merged(est, prob, logz):
    """Posterior-weighted back-rotated photons over back-rotated weights."""
    case, size = est.case, est.case['size']
    r, npix = case['rot'], size * size
    x, y = _axes(size)
    cs, sn = _rotation_angles(case)
    out = torch.zeros((len(est.params), npix), dtype=_F8, device='cuda')
    for i in range(len(est.params)):
        p = torch.exp(prob[i * r:(i + 1) * r] - logz[None])
        p = torch.where(p >= 1.e-6, p, torch.zeros_like(p))
        view, wts = p @ est.k, p @ est.scales
        num = torch.zeros(npix, dtype=_F8, device='cuda')
        den = torch.zeros(npix, dtype=_F8, device='cuda')
        base, fx, fy, ok = _footprint(size, cs, sn, x[None], y[None])
        for o, wt in _corners(fx, fy, size):
            wt = torch.where(ok, wt, torch.zeros_like(wt))
            num.index_add_(0, (base + o).view(-1), (view * wt).view(-1))
            den.index_add_(0, (base + o).view(-1), (wts[:, None] * wt).view(-1))
        out[i] = torch.where(den > 0, num / torch.where(den > 0, den, 1.), torch.zeros_like(num))
    return out


def _phaser_masks(size):
    # on the host: the masks' edges depend on the exact quotients
    ind = (np.arange(size, dtype='f8') - size // 2) / size
    qx, qy = (a.ravel() for a in np.meshgrid(ind, ind, indexing='ij'))
    q = np.sqrt(qx * qx + qy * qy)
    q[q == 0] = 1.e-6
    t = lambda a: torch.as_tensor(a).cuda()  # noqa: E731
    return t(qx), t(qy), t(q), t((q > 4 / size) & (q < 0.5)), t((q > 0.39) & (q < 0.41))


def _reference(q, th, dia):
    ff = _sphere(np.pi * q * dia)
    return ff * torch.cos(th), ff * torch.sin(th)


def _exact_phaser(case, counts, model, sx, sy, dia, ang):
    """Ring pass, mean rescale and main pass of the pattern search."""
    size, n = case['size'], counts.shape[0]
    qx, qy, q, mask, rmask = _phaser_masks(size)
    states, fs = np.unique(np.stack([sx, sy, dia], 1), axis=0, return_inverse=True)
    fs = torch.as_tensor(fs.ravel()).cuda()
    c = torch.as_tensor(np.cos(-ang)).cuda()[:, None]
    s = torch.as_tensor(np.sin(-ang)).cuda()[:, None]
    rows = torch.nonzero(mask | rmask).view(-1)
    hist = torch.zeros((len(states), rows.numel()), dtype=_F8, device='cuda')
    for lo in range(0, n, 64):
        hi = min(n, lo + 64)
        a, b = c[lo:hi], s[lo:hi]
        ux = torch.round((a * qx[rows] + (-b) * qy[rows]) * size + size // 2)
        uy = torch.round((b * qx[rows] + a * qy[rows]) * size + size // 2)
        u = (ux * size + uy).long()
        on = (u >= 0) & (u < size * size)
        k = torch.gather(counts[lo:hi].double(), 1, torch.where(on, u, 0))
        hist.index_add_(0, fs[lo:hi], torch.where(on, k, torch.zeros_like(k)))
    weight = torch.bincount(fs, minlength=len(states)).double() / n
    st = torch.as_tensor(states).cuda()
    row_of = torch.full((size * size,), -1, dtype=torch.int64, device='cuda')
    row_of[rows] = torch.arange(rows.numel(), device='cuda')
    step0 = torch.arange(33, dtype=_F8, device='cuda') * 0.5 - 8.
    pr, pi = step0[:, None].expand(33, 33).reshape(-1), step0[None].expand(33, 33).reshape(-1)
    f = torch.as_tensor(np.array(model)).cuda().clone()

    def search(pix, rescale):
        out = f[pix].clone()
        scales = torch.empty(pix.numel(), dtype=_F8, device='cuda')
        for lo in range(0, pix.numel(), 4096):
            t = pix[lo:lo + 4096]
            th = 2. * np.pi * (qx[t][None] * st[:, :1] + qy[t][None] * st[:, 1:2])
            rr, ri = _reference(q[t][None], th, st[:, 2:3])
            k = hist[:, row_of[t]]
            kmean = k.sum(0) / n
            ar, ai = (weight[:, None] * rr).sum(0), (weight[:, None] * ri).sum(0)
            var = (weight[:, None] * ((rr - ar) ** 2 + (ri - ai) ** 2)).sum(0)
            z = out[lo:lo + 4096]
            step, live = z.abs() / 4., torch.ones(t.numel(), dtype=torch.bool, device='cuda')
            used = torch.nonzero(k.sum(1) > 0).view(-1).tolist()
            for _ in range(10):
                fr, fi = z.real[:, None] + pr * step[:, None], z.imag[:, None] + pi * step[:, None]
                mw = (fr + ar[:, None]) ** 2 + (fi + ai[:, None]) ** 2 + var[:, None]
                rho = kmean[:, None] / mw if rescale is None else torch.full_like(mw, rescale)
                acc = torch.zeros_like(mw)
                for j in used:
                    w = (fr + rr[j][:, None]) ** 2 + (fi + ri[j][:, None]) ** 2
                    acc += torch.special.xlogy(k[j][:, None].expand_as(w), rho * w)
                val = acc / n - rho * mw
                if rescale is None:   # 0 log 0 in every frame: the first candidate
                    val[kmean == 0] = 0.
                best = val.argmax(1)
                zn = torch.complex(torch.gather(fr, 1, best[:, None])[:, 0],
                                   torch.gather(fi, 1, best[:, None])[:, 0])
                sn = torch.where(best == 544, step / 6.6, step)
                live = live & ~(sn / zn.abs() < 1.e-3)
                z, step = torch.where(live, zn, z), torch.where(live, sn, step)
            out[lo:lo + 4096] = z
            scales[lo:lo + 4096] = kmean / ((z.real + ar) ** 2 + (z.imag + ai) ** 2 + var)
        f[pix] = out
        return scales.mean()

    rescale = float(search(torch.nonzero(rmask).view(-1), None))
    search(torch.nonzero(mask).view(-1), rescale)
    return f.cpu().numpy()


def _accumulate(case, data, leaves, frame_loss):
    """Loss and gradients summed over blocks of frames."""
    size, n = case['size'], case['frames']
    k = _counts(case, data, torch.float32)
    leaves = [v.double().clone().requires_grad_(True) for v in leaves]
    total = 0.
    block = max(16, int(2e6 / size ** 2))
    for lo in range(0, n, block):
        hi = min(n, lo + block)
        loss = frame_loss(slice(lo, hi), k[lo:hi].double(), *leaves)
        loss.backward()
        total += float(loss.detach())
    return dict(loss=torch.tensor(total, dtype=_F8), grads=[v.grad for v in leaves])


def _exact_nll(case, data, model):
    size = case['size']
    qx, qy, q, mask, _ = _phaser_masks(size)
    pix = torch.nonzero(mask).view(-1)
    qx, qy, q = qx[pix], qy[pix], q[pix]
    ang = -np.asarray(data['true_angles'])
    c, s = torch.as_tensor(np.cos(ang)).cuda()[:, None], torch.as_tensor(np.sin(ang)).cuda()[:, None]

    def frame_loss(sl, k, fre, fim, dia, sx, sy, scale):
        ux = torch.round((c[sl] * qx + (-s[sl]) * qy) * size + size // 2)
        uy = torch.round((s[sl] * qx + c[sl] * qy) * size + size // 2)
        u = (ux * size + uy).long()
        on = (ux >= 0) & (ux < size) & (uy >= 0) & (uy < size)
        kt = torch.where(on, torch.gather(k, 1, torch.where(on, u, 0)), 0.)
        th = 2. * np.pi * (qx * sx[sl, None] + qy * sy[sl, None])
        rr, ri = _reference(q[None], th, dia[sl, None])
        w = scale[sl, None] * ((fre + rr) ** 2 + (fim + ri) ** 2)
        return (w - kt * torch.log(w)).sum()

    return _accumulate(case, data, _leaves(case, data, model[pix.cpu().numpy()]), frame_loss)


def _exact_slice_nll(case, data, model):
    from rspi import geometry
    size = case['size']
    sel = _likelihood_pixels(size)
    x, y = _axes(size)
    r = torch.sqrt(x * x + y * y)
    vscale = _vscale(case, data, model, geometry.emc_masks(size)[1])
    ang = np.asarray(data['true_angles'])
    c, s = torch.as_tensor(np.cos(ang)).cuda()[:, None], torch.as_tensor(np.sin(ang)).cuda()[:, None]

    def frame_loss(sl, k, mre, mim, dia, sx, sy, scale):
        sv = r[None] * np.pi * dia[sl, None] / size
        ff = _sphere(torch.where(sv == 0., torch.full_like(sv, 1.e-5), sv))
        th = 2. * np.pi * (x * sx[sl, None] + y * sy[sl, None]) / size
        w = (torch.cos(th) * ff + mre) ** 2 + (torch.sin(th) * ff + mim) ** 2
        base, fx, fy, ok = _footprint(size, c[sl], s[sl], x[sel][None], y[sel][None])
        v = sum(torch.gather(w, 1, base + o) * wt for o, wt in _corners(fx, fy, size))
        bad = ~ok | (v < 1.e-20)
        lv = torch.where(bad, torch.full_like(v, -1000.), torch.log(torch.where(bad, 1., v)))
        ks = k[:, sel]
        return (vscale * scale[sl] * w[:, sel].sum(1)).sum() - \
            (ks * (torch.log(scale[sl, None]) + lv)).sum()

    return _accumulate(case, data, _leaves(case, data, model), frame_loss)


def _exact_refine(case, model):
    size = case['size']
    x, y = _axes(size)
    r = torch.sqrt(x * x + y * y).view(size, size)
    f = torch.as_tensor(model).cuda().view(size, size)
    fwd = lambda a: torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(a)))  # noqa: E731
    inv = lambda a: torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(a)))  # noqa: E731
    sm = inv(f * torch.special.expit((r - 12.) / 2.)).real.abs()
    w = torch.exp(-0.5 / 9. * torch.arange(-12, 13, dtype=_F8, device='cuda') ** 2)
    w = w / w.sum()
    for axis in (0, 1):
        a = sm.movedim(axis, 1)
        a = torch.cat([a[:, :12].flip(1), a, a[:, -12:].flip(1)], 1)
        sm = sum(w[i] * a[:, i:i + size] for i in range(25)).movedim(1, axis)
    outside = ~(sm > 1.2e-4)
    known = (r >= 4) & (r < size // 2)

    def real(z):
        z = inv(z).real
        return fwd(torch.where((z < 0) | outside, torch.zeros_like(z), z).to(torch.complex128))

    v = f
    for _ in range(10):
        p1 = torch.where(known, f, v)
        v = v + real(2. * p1 - v) - p1
    for _ in range(5):
        v = real(torch.where(known, f, v))
    return v.reshape(-1)


def exact(case, seed):
    data, model = _data(case, seed)
    kind, n0 = case['kind'], case['shifts'] ** 2 * case['dias']
    if kind in ('iterate', 'posterior', 'fp64', 'dense'):
        est = _ExactEStep(case, data, model)
        best, arg, logz, prob = est.reduce(kind != 'iterate')
        if kind == 'iterate':
            arg = arg.cpu().numpy()
            mode, state = arg // (n0 * case['rot']), arg // case['rot'] % n0
            vals = np.array(est.values)[state]
            ang = arg % case['rot'] * np.pi / case['rot']
            counts = est.k.float()
            del est
            models = np.array(model).reshape(case['modes'], -1)
            for m in range(case['modes']):
                mine = np.flatnonzero(mode == m)
                if mine.size:
                    models[m] = _exact_phaser(case, counts[torch.as_tensor(mine).cuda()],
                                              models[m], vals[mine, 0], vals[mine, 1],
                                              vals[mine, 2], ang[mine])
            return dict(model=models.reshape(model.shape), rmax=arg.astype('i4'))
        out = dict(maxll=best, rmax=arg.int(), logz=logz, prob=prob)
        if kind == 'posterior':
            out['intens'] = _merged(est, prob, logz)
        return out
    if kind == 'phaser':
        return _exact_phaser(case, _counts(case, data, torch.float32), model,
                             *_nearest_states(case, data))
    if kind == 'nll':
        return _exact_nll(case, data, model)
    if kind == 'slicenll':
        return _exact_slice_nll(case, data, model)
    return _exact_refine(case, model)
