"""Workloads of the pair-binning library as its users run them.

Each case is one call of the public entry points on a synthetic catalogue of
one of the repository's configurations (``lya2pcf_b200/synthetic.py``: sky
density, forest lengths and windows as documented there):

* ``corr``  -- catalogue resident on the GPU: neighbour search, per-pixel
  histograms, copy-out (the step of ``bench.py``); FP32-guarded or FP64 kernel.
* ``ingest`` -- the same from host arrays: upload of the deltas, device
  projection, neighbour search, histograms, copy-out (a new catalogue or a
  new mock with an engine that is kept).
* ``grad``  -- one step of a fit: projection of the deltas, xi and the
  gradient of a loss with respect to the weights and the deltas.
* ``dist``  -- distortion matrix of the work queue (one owner pixel, or a patch).
* ``cov``   -- covariance and its smoothing from the per-pixel files' arrays.
* ``covrun`` -- the same from the histograms that a run left on the device.
"""
import math

import numpy as np
import torch

from lya2pcf_b200 import _native, autograd, covariance, synthetic
from lya2pcf_b200.engine import PairEngine

RMAX = 200.0
PAIR_FLOPS = 17.0      # geometry and five sums of one pixel pair
GRAD_FLOPS = 8.0       # two products for either pixel of a pair
DIST_FLOPS = 2.3e7     # block products of one forest pair at 50 x 50 bins


def _corr(name, config, n, kernel='fp32', np_=50, nt=50):
    return dict(name=name, kind='corr', config=config, n=n, kernel=kernel, np=np_, nt=nt)


def listed():
    return [
        # a 10 deg^2 field: one call is latency, launches and a short kernel
        _corr('corr_500', 4, 500),
        # a 100 deg^2 field with long forests
        _corr('corr_2000', 0, 2000),
        # a slice of a survey, 640 deg^2: the throughput of the pair kernel
        _corr('corr_12000', 1, 12000),
        # the FP64 kernel, taken for cross-checks, with an odd binning
        _corr('corr_fp64_odd', 0, 1500, 'fp64', 37, 23),
        # new data on a kept engine: 220 deg^2 of deltas from the host
        dict(name='ingest_4000', kind='ingest', config=1, n=4000, np=50, nt=50),
        # one step of a fit in double precision on a small field
        dict(name='grad_500_f64', kind='grad', config=4, n=500, kernel='fp64', dtype='float64', np=50, nt=50),
        # the same in single precision on a larger field, FP32-guarded forward
        dict(name='grad_2500_f32', kind='grad', config=0, n=2500, kernel='fp32', dtype='float32', np=50, nt=50),
        # distortion of about one owner pixel, the unit of the distortion driver
        dict(name='dist_60', kind='dist', config=3, n=60, np=50, nt=50),
        # distortion of a clustered patch
        dict(name='dist_600', kind='dist', config=3, n=600, np=50, nt=50),
        # covariance over the owner pixels of a whole survey, from host arrays
        dict(name='cov_676', kind='cov', n=676, np=50, nt=50),
        # covariance of a run, straight from the device
        dict(name='covrun_1000', kind='covrun', config=0, n=1000, np=30, nt=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['corr', 'corr', 'corr', 'ingest', 'grad', 'grad', 'dist', 'dist', 'cov', 'covrun'])
    np_, nt = rng.choice([(50, 50), (50, 50), (50, 50), (40, 40), (37, 23), (25, 25), (64, 32)])
    case = dict(kind=kind, np=np_, nt=nt)
    if kind == 'corr':
        case['kernel'] = rng.choice(['fp32', 'fp32', 'fp64'])
        case['config'] = rng.choice([0, 1, 4])
        case['n'] = _log_int(rng, 200, 1800 if case['kernel'] == 'fp64' else {0: 3500, 1: 11000, 4: 4500}[case['config']])
    elif kind == 'ingest':
        case['config'] = rng.choice([0, 1])
        case['n'] = _log_int(rng, 300, 3500 if case['config'] else 2000)
    elif kind == 'grad':
        case['kernel'], case['dtype'] = rng.choice([('fp64', 'float64'), ('fp64', 'float32'), ('fp32', 'float32')])
        case['config'] = rng.choice([0, 4])
        case['n'] = _log_int(rng, 200, 1500)
    elif kind == 'dist':
        case['config'] = rng.choice([3, 3, 4])
        case['n'] = _log_int(rng, 40, 500 if case['config'] == 3 else 200)
    elif kind == 'cov':
        case['np'], case['nt'] = rng.choice([(50, 50), (40, 40), (25, 25)])
        case['n'] = _log_int(rng, 48, 1000)
    else:
        # every bin needs pairs of several owner pixels, or its variance is rounding noise
        case['np'], case['nt'] = rng.choice([(25, 25), (30, 30), (30, 20)])
        case['config'], case['n'] = 0, _log_int(rng, 700, 1800)
    return case


KERNELS = {'fp32': _native.KERNEL_FP32_GUARDED, 'fp64': _native.KERNEL_FP64_DIAGONAL}


def _catalogue(case, seed):
    """A mock of the configuration's survey: forest lengths, windows and owner
    pixels are the survey's; weights, deltas, sky positions (moved by up to 2
    arcminutes) and the distance scale (a fit's cosmology, within 1%) the seed's."""
    fs = synthetic.make(case['config'], n=case['n'])
    rng = np.random.default_rng(seed)
    fs.dc = fs.dc * rng.uniform(0.99, 1.01)
    fs.ra = fs.ra + rng.uniform(-6e-4, 6e-4, fs.n)
    fs.dec = fs.dec + rng.uniform(-6e-4, 6e-4, fs.n)
    fs.ux, fs.uy, fs.uz = np.cos(fs.ra) * np.cos(fs.dec), np.sin(fs.ra) * np.cos(fs.dec), np.sin(fs.dec)
    lengths = fs.lengths
    mean = lambda v: np.add.reduceat(v, fs.start[:-1])  # noqa: E731
    fs.w = ((1.0 + fs.z) / 3.25) ** 1.9 / (0.1 + rng.uniform(0.01, 0.5, fs.npix_total))
    delta, loglam = _deltas(fs, seed)
    fs.omega = mean(fs.w)
    fs.dl = loglam - np.repeat(mean(fs.w * loglam) / fs.omega, lengths)
    fs.odl2 = mean(fs.w * fs.dl ** 2)
    slope = mean(fs.w * fs.dl * delta) / fs.odl2
    fs.dw = fs.w * (delta - np.repeat(mean(fs.w * delta) / fs.omega, lengths) - fs.dl * np.repeat(slope, lengths))
    return fs


def _deltas(fs, seed):
    """log10(lambda) of every pixel, and deltas before the projection."""
    loglam = np.log10((1.0 + fs.z) * 1215.67)
    delta = np.random.default_rng(seed + 1).normal(0.0, synthetic.SIGMA_DELTA, fs.npix_total)
    return delta, loglam


def _cov_inputs(case, seed):
    """Correlation estimates and weights of n owner pixels in nb bins."""
    rng = np.random.default_rng(seed)
    nb = case['np'] * case['nt']
    w = rng.uniform(0.5, 3.0, (case['n'], 1)) * rng.uniform(1e3, 1e4, (1, nb)) * rng.uniform(0.7, 1.3, (case['n'], nb))
    xi = 1e-4 * rng.standard_normal((case['n'], nb)) + 1e-5 * rng.standard_normal((case['n'], 1))
    return xi, w


def prepare(case, seed):
    kind = case['kind']
    if kind == 'cov':
        xi, w = _cov_inputs(case, seed)
        return dict(case=case, xi=xi, w=w, bins=covariance.bin_coordinates(case['np'], case['nt']))
    fs = _catalogue(case, seed)
    state = dict(case=case, fs=fs, angmax=synthetic.angmax_for(fs, RMAX))
    eng = state['eng'] = PairEngine(0, RMAX, RMAX, case['np'], case['nt'])
    if kind == 'ingest':
        state['delta'], state['loglam'] = _deltas(fs, seed)
        return state
    eng.upload(fs)
    if kind == 'grad':
        eng.build_pairs(state['angmax'])
        dtype = getattr(torch, case['dtype'])
        delta, loglam = _deltas(fs, seed)
        state['w'] = torch.tensor(fs.w, dtype=dtype, device='cuda').requires_grad_()
        state['delta'] = torch.tensor(delta, dtype=dtype, device='cuda').requires_grad_()
        state['loglam'] = torch.tensor(loglam, dtype=dtype, device='cuda')
        state['fid'] = autograd.forest_index(fs.start, 'cuda')
        state['g'] = torch.tensor(np.random.default_rng(seed + 2).standard_normal(eng.nb), dtype=dtype, device='cuda')
    elif kind in ('dist', 'covrun'):
        eng.build_pairs(state['angmax'])
        if kind == 'covrun':
            eng.run(kernel=_native.KERNEL_FP64_DIAGONAL)
    return state


def run(state):
    case, kind = state['case'], state['case']['kind']
    if kind == 'cov':
        c, mean = covariance.cov(state['xi'], state['w'], numpix=(case['np'], case['nt']))
        smooth = covariance.cov_smooth(state['xi'], state['w'], *state['bins'], c, numpix=(case['np'], case['nt']))
        return dict(mean=mean, cov=c, smooth=smooth)
    eng = state['eng']
    if kind == 'covrun':
        mean, c, smooth, _ = eng.covariance()
        return dict(mean=mean, cov=c, smooth=smooth)
    if kind == 'dist':
        D, W = eng.distortion()
        return dict(D=D, W=W)
    if kind == 'grad':
        w, delta = state['w'], state['delta']
        dw = autograd.project_delta(w, delta, state['loglam'], state['fid'], state['fs'].n)
        xi = autograd.xi(w, dw, eng, kernel=KERNELS[case['kernel']])
        gw, gdelta = torch.autograd.grad((state['g'] * xi).sum(), (w, delta))
        return dict(xi=xi.detach(), gw=gw, gdelta=gdelta)
    if kind == 'ingest':
        eng.upload_deltas(state['fs'], state['delta'], state['loglam'])
    eng.build_pairs(state['angmax'])
    eng.run(kernel=KERNELS[case.get('kernel', 'fp32')])
    hist, counts = eng.histograms()
    return dict(hist=hist, counts=counts)


# ------------------------------------------------------------------ what a pass cannot do without
def _estimate(case):
    """(forest pairs, pixel pairs in range, pixels) of a case, from its sky density and lengths."""
    cfg = synthetic.CONFIGS[case['config']]
    n = case['n']
    ra0, ra1 = cfg['ra']
    d0, d1 = cfg['dec']
    mid = math.cos(math.radians(0.5 * (d0 + d1)))
    width, height, theta = (ra1 - ra0) * n / cfg['n'] * mid, d1 - d0, 3.2
    density = n / (width * height)
    reach = math.pi * theta ** 2 * min(1.0, width / (1.6 * theta)) * min(1.0, height / (1.6 * theta))
    pairs = min(0.5 * n * (n - 1), 0.5 * n * density * reach)
    length = 0.5 * (cfg['length'][0] + min(cfg['length'][1], synthetic.NGRID))
    return pairs, pairs * 0.28 * length ** 2, n * length


def work(case):
    nb = case['np'] * case['nt']
    if case['kind'] == 'cov':
        n = case['n']
        return dict(bytes=16.0 * n * nb + 16.0 * nb * nb, flops=float(n) * nb * nb)
    pairs, pixel_pairs, pixels = _estimate(case)
    slots = max(1.0, case['n'] / 250.0)
    if case['kind'] == 'covrun':
        return dict(bytes=16.0 * slots * nb + 16.0 * nb * nb, flops=slots * nb * nb)
    if case['kind'] == 'dist':
        return dict(bytes=24.0 * pixels + 8.0 * nb * nb, flops=pairs * DIST_FLOPS * (nb / 2500.0) * (pixels / case['n'] / 332.0))
    if case['kind'] == 'grad':
        item = 8 if case['dtype'] == 'float64' else 4
        return dict(bytes=(5.0 * item + 8.0) * pixels, flops=pixel_pairs * (PAIR_FLOPS + GRAD_FLOPS))
    bytes_ = 32.0 * pixels + 48.0 * slots * nb + (40.0 * pixels if case['kind'] == 'ingest' else 0.0)
    return dict(bytes=bytes_, flops=pixel_pairs * PAIR_FLOPS)


# ------------------------------------------------------------------ 64-bit values, plain torch
def _neighbours(fs, angmax):
    t = lambda a: torch.tensor(a, device='cuda')  # noqa: E731
    x, y, z, ra, name = t(fs.ux), t(fs.uy), t(fs.uz), t(fs.ra), t(fs.name)
    mu = (x[:, None] * x + y[:, None] * y) + z[:, None] * z
    near = (mu > math.cos(angmax)) & (ra[:, None] < ra) & (name[:, None] != name)
    f1, f2 = near.nonzero(as_tuple=True)
    return f1, f2, mu


def _blocks(fs, angmax, np_, nt, most=1 << 25):
    """Forest pairs in blocks of equal padded shape: pixel indices i, j (padding:
    the index past the last pixel), the flat bin of every pair (nb: none), rp, rt."""
    f1, f2, mu = _neighbours(fs, angmax)
    start = torch.tensor(fs.start, device='cuda')
    dc = torch.cat([torch.tensor(fs.dc, device='cuda'), torch.full((1,), math.inf, dtype=torch.float64, device='cuda')])
    length = start[1:] - start[:-1]
    top = int(length.max())
    k = torch.arange(top, device='cuda')
    at = torch.where(k < length[:, None], start[:-1, None] + k, fs.npix_total)
    for c in range(0, len(f1), max(1, most // top ** 2)):
        a, b = f1[c:c + max(1, most // top ** 2)], f2[c:c + max(1, most // top ** 2)]
        i, j, m = at[a], at[b], mu[a, b].clamp(-1.0, 1.0)
        d1, d2 = dc[i][:, :, None], dc[j][:, None, :]
        rp = (d1 - d2).abs() * torch.sqrt(0.5 * (1.0 + m))[:, None, None]
        rt = (d1 + d2) * torch.sqrt(0.5 * (1.0 - m))[:, None, None]
        bp, bt = torch.floor(rp * (np_ / RMAX)), torch.floor(rt * (nt / RMAX))
        ok = (bp < np_) & (bt < nt)
        flat = torch.where(ok, bp * nt + bt, float(np_ * nt)).nan_to_num(float(np_ * nt)).long()
        yield a, b, i, j, flat, rp, rt


def _padded(v):
    return torch.cat([torch.as_tensor(v, dtype=torch.float64, device='cuda').detach(), torch.zeros(1, dtype=torch.float64, device='cuda')])


def _project(w, delta, loglam, fid, n):
    seg = lambda v: torch.zeros(n, dtype=v.dtype, device=v.device).index_add(0, fid, v)  # noqa: E731
    sw = seg(w)
    dl = loglam - (seg(w * loglam) / sw)[fid]
    slope = seg(w * dl * delta) / seg(w * dl * dl)
    return w * (delta - (seg(w * delta) / sw)[fid] - dl * slope[fid])


def _exact_corr(case, fs, dw):
    np_, nt = case['np'], case['nt']
    nb = np_ * nt
    pix = fs.pix
    slot = torch.tensor(np.cumsum(np.concatenate([[0], pix[1:] != pix[:-1]])), device='cuda')
    w, dw, z = _padded(fs.w), _padded(dw), _padded(fs.z)
    hist = torch.zeros(int(slot[-1]) + 1, 5, nb + 1, dtype=torch.float64, device='cuda')
    for a, b, i, j, flat, rp, rt in _blocks(fs, synthetic.angmax_for(fs, RMAX), np_, nt):
        ww = w[i][:, :, None] * w[j][:, None, :]
        rp, rt = rp.nan_to_num(0.0, 0.0), rt.nan_to_num(0.0, 0.0)
        sums = (ww, dw[i][:, :, None] * dw[j][:, None, :], ww * rp, ww * rt, ww * 0.5 * (z[i][:, :, None] + z[j][:, None, :]))
        for s in slot[a].unique().tolist():
            own = slot[a] == s
            for q, v in enumerate(sums):
                hist[s, q] += torch.bincount(flat[own].reshape(-1), weights=v[own].reshape(-1), minlength=nb + 1)
    return dict(hist=hist[:, :, :nb].contiguous(), counts=None)


def _exact_grad(case, fs, seed):
    np_, nt = case['np'], case['nt']
    nb = np_ * nt
    dtype = getattr(torch, case['dtype'])
    given = lambda a: torch.tensor(a, device='cuda').to(dtype).double()  # noqa: E731
    delta, loglam = (given(a) for a in _deltas(fs, seed))
    w, g = given(fs.w).requires_grad_(), given(np.random.default_rng(seed + 2).standard_normal(nb))
    delta.requires_grad_()
    fid = autograd.forest_index(fs.start, 'cuda')
    dw = _project(w, delta, loglam, fid, fs.n)
    pw, pdw = _padded(w), _padded(dw)
    tot = torch.zeros(2, nb + 1, dtype=torch.float64, device='cuda')
    angmax = synthetic.angmax_for(fs, RMAX)
    for a, b, i, j, flat, rp, rt in _blocks(fs, angmax, np_, nt):
        for q, v in enumerate((pw, pdw)):
            tot[q] += torch.bincount(flat.reshape(-1), weights=(v[i][:, :, None] * v[j][:, None, :]).reshape(-1), minlength=nb + 1)
    W, DW = tot[0, :nb], tot[1, :nb]
    xi = torch.where(W != 0, DW / torch.where(W != 0, W, 1.0), 0.0)
    per_w = torch.where(W != 0, g / torch.where(W != 0, W, 1.0), 0.0)
    table = [torch.cat([t, torch.zeros(1, dtype=torch.float64, device='cuda')]) for t in (per_w, -per_w * xi)]
    grads = [torch.zeros_like(pw) for _ in range(2)]
    for a, b, i, j, flat, rp, rt in _blocks(fs, angmax, np_, nt):
        for out, v, t in zip(grads, (pdw, pw), table):
            c = t[flat]
            out.index_add_(0, i.reshape(-1), (c * v[j][:, None, :]).sum(2).reshape(-1))
            out.index_add_(0, j.reshape(-1), (c * v[i][:, :, None]).sum(1).reshape(-1))
    gdw, gw = grads[0][:-1], grads[1][:-1]
    from_dw = torch.autograd.grad(dw, (w, delta), gdw)
    return dict(xi=xi, gw=gw + from_dw[0], gdelta=from_dw[1])


def _exact_dist(case, fs):
    np_, nt = case['np'], case['nt']
    nb = np_ * nt
    D = torch.zeros(nb + 1, nb + 1, dtype=torch.float64, device='cuda')
    W = torch.zeros(nb + 1, dtype=torch.float64, device='cuda')
    w, dl = _padded(fs.w), _padded(fs.dl)
    om, o2 = torch.tensor(fs.omega, device='cuda'), torch.tensor(fs.odl2, device='cuda')
    for a, b, i, j, flat, rp, rt in _blocks(fs, synthetic.angmax_for(fs, RMAX), np_, nt):
        for p in range(len(a)):
            bins, at = flat[p].unique(return_inverse=True)
            nA, L1, L2 = len(bins), i.shape[1], j.shape[1]
            wi, li, wj, lj = w[i[p]], dl[i[p]], w[j[p]], dl[j[p]]
            def columns(v, side):   # sum over the other forest's pixels of each bin
                out = torch.zeros(nA, L1 if side == 0 else L2, dtype=torch.float64, device='cuda')
                rows = torch.arange(out.shape[1], device='cuda')
                where = (at, rows[:, None].expand(L1, L2)) if side == 0 else (at, rows[None, :].expand(L1, L2))
                return out.index_put_(where, (v[None, :] if side == 0 else v[:, None]).expand(L1, L2), accumulate=True)
            S2, K2, S1, K1 = columns(wj, 0), columns(wj * lj, 0), columns(wi, 1), columns(wi * li, 1)
            m0, mi, mj, mij = S2 @ wi, S2 @ (wi * li), K2 @ wi, K2 @ (wi * li)
            n1, n2, q1, q2 = om[a[p]], om[b[p]], o2[a[p]], o2[b[p]]
            block = torch.diag(m0) + torch.outer(m0, m0) / (n1 * n2) + torch.outer(mj, mj) / (n1 * q2) \
                + torch.outer(mi, mi) / (q1 * n2) + torch.outer(mij, mij) / (q1 * q2) \
                - (S2 * wi) @ S2.T / n2 - (K2 * wi) @ K2.T / q2 - (S1 * wj) @ S1.T / n1 - (K1 * wj) @ K1.T / q1
            D[bins[:, None], bins[None, :]] += block
            W[bins] += m0
    return dict(D=D[:nb, :nb].contiguous(), W=W[:nb].contiguous())


def _exact_cov(case, seed):
    xi, w = (torch.tensor(v, device='cuda') for v in _cov_inputs(case, seed))
    W = w.sum(0)
    mean = (xi * w).sum(0) / W
    y = w * (xi - mean)
    c = (y.T @ y) / torch.outer(W, W)
    sd = c.diagonal().sqrt()
    corr = c / torch.outer(sd, sd)
    rp, rt = (torch.tensor(v, device='cuda') for v in covariance.bin_coordinates(case['np'], case['nt']))
    step = ((rp[:, None] - rp).abs() * case['nt'] + (rt[:, None] - rt).abs()).reshape(-1)
    upper = torch.ones_like(c).triu(1).reshape(-1)
    total = torch.bincount(step, weights=corr.reshape(-1) * upper)
    count = torch.bincount(step, weights=upper)
    smooth = (total / count)[step].reshape(c.shape) * torch.outer(sd, sd)
    smooth.diagonal().copy_(c.diagonal())
    return dict(mean=mean, cov=c, smooth=smooth)


def exact(case, seed):
    kind = case['kind']
    if kind == 'cov':
        return _exact_cov(case, seed)
    pairs, pixel_pairs, _ = _estimate(case)
    if kind == 'covrun' or pixel_pairs > 4e9 or (kind == 'dist' and pairs > 4000):
        return None
    fs = _catalogue(case, seed)
    if kind == 'dist':
        return _exact_dist(case, fs)
    if kind == 'grad':
        return _exact_grad(case, fs, seed)
    if kind == 'ingest':
        delta, loglam = (torch.tensor(v, device='cuda') for v in _deltas(fs, seed))
        fid = torch.tensor(np.repeat(np.arange(fs.n), fs.lengths), device='cuda')
        return _exact_corr(case, fs, _project(torch.tensor(fs.w, device='cuda'), delta, loglam, fid, fs.n))
    return _exact_corr(case, fs, torch.tensor(fs.dw, device='cuda'))
