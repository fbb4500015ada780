"""The framework's measured work: exact F(Q), its gradient, the PDF potential
and the samplers, through the public entry points, from one small cluster to
the 20,000-atom particle of the benchmark.

``listed()`` are the standing cases, ``draw(rng)`` gives others of the same
ranges, ``prepare(case, seed)`` builds what a program holds before the call,
``run(state)`` is one pass, ``work(case)`` what a pass cannot do without, and
``exact(case, seed)`` the outputs in 64 bits from plain torch and numpy.

Particles are fcc lattices with seeded thermal displacements (0.02-0.05 A),
elements mixed at random, atoms in the order of their distance from the
centre: what a structure refinement starts from.  The Q and r grids are the
ones of the benchmark, the tests and the reference's defaults.
"""
import functools
import math

import numpy as np
import torch

from pyiid_gb300 import debye, structures
from pyiid_gb300.sampling import (BatchedHMC, PDFPotential, SingleAtomMC,
                                  experiment_grids)
from pyiid_gb300.scatter_factors import form_factor_array

# F(Q) grids: Q step, bins from Q = 0, first returned bin
GRIDS = {
    'default': (0.1, 250, 0),     # the reference's defaults: qmax 25, qbin 0.1
    'fine': (0.05, 500, 2),       # Q 0.1-25 step 0.05
    'high': (0.02, 1500, 25),     # Q 0.5-30 step 0.02
}
ELEMENTS = (79, 78, 46)           # Au, Pt, Pd


def listed():
    return [
        # the smallest call: F(Q) of one cluster, get_fq of a first look at a
        # structure; launches and host work are all there is
        dict(name='fq_au55', kind='fq', n=55, species=1, grid='default'),
        # one evaluation of F(Q) with its gradient at the size of the
        # reference's own benchmark particle
        dict(name='fq_grad_au249', kind='fq_grad', n=249, species=1,
             grid='fine'),
        # the same for the particle that the samplers run on
        dict(name='fq_grad_au1000', kind='fq_grad', n=1000, species=1,
             grid='fine'),
        # get_grad_fq of a drop-in calculator on an alloy, ragged in atoms
        # and bins (2,001 atoms, 1,475 returned bins)
        dict(name='grad_fq_alloy2001', kind='grad_fq', n=2001, species=2,
             grid='high'),
        # the benchmark's step: F(Q) and the whole gradient of 20,000 atoms
        dict(name='fq_grad_au20000', kind='fq_grad', n=20000, species=1,
             grid='high'),
        # F(Q) alone of a large particle: a forward model without a fit
        dict(name='fq_au10007', kind='fq', n=10007, species=1, grid='high'),
        # many alloys of uneven sizes in one call: a library of structures
        # compared with one measurement
        dict(name='batch_fq_alloys256', kind='batch_fq', configs=256,
             n_min=55, n_max=2000, species=2, grid='fine'),
        # Rw and its gradient of one particle: each step of a refinement
        dict(name='potential_au309', kind='potential', configs=1, n=309,
             species=1, potential='rw', gradient=True, rmax=40.0),
        # the same for 64 chains at once: each leapfrog step of batched HMC
        dict(name='potential_au1000x64', kind='potential', configs=64, n=1000,
             species=1, potential='rw', gradient=True, rmax=40.0),
        # a whole sampler call: one HMC iteration (10 leapfrog steps and the
        # acceptance) of 16 chains, replayed as the CUDA graph it captures
        dict(name='hmc_au309x16', kind='hmc', configs=16, n=309,
             species=1, leapfrog=10),
        # G(r) gradient of every atom from the gradient of F(Q): the drop-in
        # get_grad_pdf
        dict(name='grad_pdf_au1000', kind='grad_pdf', n=1000, rmax=40.0),
        # single-atom Metropolis: 16 proposals of each of 64 chains
        dict(name='mh_au1000x64', kind='mh', configs=64, n=1000, species=1,
             steps=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fq', 'fq_grad', 'fq_grad', 'grad_fq', 'batch_fq',
                       'potential', 'potential', 'hmc', 'grad_pdf', 'mh'])
    species = rng.choice([1, 1, 2, 3])
    if kind in ('fq', 'fq_grad', 'grad_fq'):
        return dict(kind=kind, n=_log_int(rng, 20, 20000), species=species,
                    grid=rng.choice(sorted(GRIDS)))
    if kind == 'batch_fq':
        lo = _log_int(rng, 2, 300)
        return dict(kind=kind, configs=_log_int(rng, 2, 256), n_min=lo,
                    n_max=lo + _log_int(rng, 1, 1700), species=species,
                    grid=rng.choice(['default', 'fine']))
    rmax = rng.choice([20.0, 30.0, 40.0])
    if kind == 'grad_pdf':
        return dict(kind=kind, n=_log_int(rng, 10, 1500), rmax=rmax)
    n = _log_int(rng, 20, 1500)
    configs = _log_int(rng, 1, 64)
    if kind == 'potential':
        return dict(kind=kind, configs=configs, n=n, species=species,
                    potential=rng.choice(['rw', 'rw', 'chi_sq']),
                    gradient=rng.choice([True, True, False]), rmax=rmax)
    if kind == 'hmc':
        return dict(kind=kind, configs=min(configs, 32), n=min(n, 1000),
                    species=species, leapfrog=rng.choice([3, 5, 10]))
    return dict(kind=kind, configs=configs, n=n, species=species,
                steps=_log_int(rng, 1, 32))


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=32)
def _sites(n):
    return structures.fcc_nearest(4.08, n)


def _numbers(rng, n, species):
    return np.asarray(ELEMENTS[:species])[rng.integers(0, species, n)]


def _table(numbers, qbin, n_bins):
    """Species ids and form factors [S, n_bins] of an atom list."""
    uniq, sp = np.unique(numbers, return_inverse=True)
    q = np.arange(n_bins) * qbin
    return (sp.reshape(-1).astype(np.int32),
            np.stack([form_factor_array(z, q) for z in uniq])
            .astype(np.float32))


def _inputs(case, seed):
    """What the seed alone decides, as host arrays."""
    rng = np.random.default_rng([int(seed), 11])
    kind = case['kind']
    if kind in ('fq', 'fq_grad', 'grad_fq'):
        n = case['n']
        qbin, n_bins, kb = GRIDS[case['grid']]
        pos = (_sites(n) + rng.normal(0, .03, (n, 3))).astype(np.float32)
        sp, tab = _table(_numbers(rng, n, case['species']), qbin, n_bins)
        return dict(pos=pos, sp=sp, tab=tab, qbin=qbin, kb=kb,
                    off=np.array([0, n], np.int32))
    if kind == 'batch_fq':
        qbin, n_bins, kb = GRIDS[case['grid']]
        # the sizes belong to the case, the structures to the seed
        sizes = np.random.default_rng(case['configs']).integers(
            case['n_min'], case['n_max'] + 1, case['configs'])
        sites = _sites(int(sizes.max()))
        pos = np.concatenate([sites[:n] + rng.normal(0, .05, (n, 3))
                              for n in sizes]).astype(np.float32)
        sp, tab = _table(_numbers(rng, len(pos), case['species']), qbin,
                         n_bins)
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
        return dict(pos=pos, sp=sp, tab=tab, qbin=qbin, kb=kb, off=off)
    if kind == 'grad_pdf':
        exp, qstep, n_bins, rgrid = experiment_grids({'rmax': case['rmax']})
        # the spread of a real gradient: thermal noise on a Q-dependent scale
        scale = (0.1 + np.arange(n_bins) * qstep) / 25.0
        g = rng.normal(0, 1, (case['n'], 3, n_bins)) * scale
        return dict(grad=g.astype(np.float32), qstep=qstep, exp=exp,
                    rgrid=rgrid)
    exp_dict = {'rmax': case.get('rmax', 40.0)}
    exp, qstep, n_bins, rgrid = experiment_grids(exp_dict)
    n, b = case['n'], case['configs']
    # chains of one particle: the same elements, other displacements
    numbers = _numbers(rng, n, case['species'])
    sites = _sites(n)
    start = (sites[None] + rng.normal(0, .05, (b, n, 3))).astype(np.float32)
    sp, tab = _table(numbers, qstep, n_bins)
    fq = _exact_fq(torch.as_tensor(sites.astype(np.float32)), sp, tab,
                   qstep, 0)
    gobs = (fq @ torch.as_tensor(_transform(case.get('rmax', 40.0)),
                                 device=fq.device)).cpu().numpy()
    return dict(start=start, numbers=numbers, gobs=gobs, exp_dict=exp_dict,
                exp=exp, qstep=qstep, rgrid=rgrid, sp=sp, tab=tab)


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = s['kind'] = case['kind']
    if kind in ('fq', 'fq_grad', 'grad_fq', 'batch_fq'):
        s['pos'] = torch.as_tensor(s['pos'], device='cuda')
    elif kind == 'grad_pdf':
        s['grad'] = torch.as_tensor(s['grad'], device='cuda')
    else:
        b = case['configs']
        pot = PDFPotential(s['numbers'], s['gobs'], s['exp_dict'],
                           potential=case.get('potential', 'rw'), conv=100.0,
                           n_configs=b)
        if kind == 'potential':
            s['pot'], s['gradient'] = pot, case['gradient']
            s['x'] = torch.as_tensor(s['start'], device='cuda').reshape(-1, 3)
        elif kind == 'hmc':
            s['hmc'] = BatchedHMC(pot, s['start'], temperature=300.0, dt=1e-3,
                                  n_steps=case['leapfrog'], seed=seed,
                                  graph=True)
        else:
            s['mc'] = SingleAtomMC(pot, s['start'], temperature=300.0,
                                   sigma=0.1, seed=seed)
            s['steps'] = case['steps']
    return s


def run(s):
    kind = s['kind']
    if kind == 'fq':
        return debye.fq(s['pos'], s['sp'], s['tab'], s['qbin'],
                        k_begin=s['kb'])
    if kind == 'fq_grad':
        return debye.fq_grad(s['pos'], s['sp'], s['tab'], s['qbin'],
                             k_begin=s['kb'])
    if kind == 'grad_fq':
        return debye.grad_fq(s['pos'], s['sp'], s['tab'], s['qbin'],
                             k_begin=s['kb'])
    if kind == 'batch_fq':
        return debye.batch_fq(s['pos'], s['sp'], s['off'], s['tab'],
                              s['qbin'], k_begin=s['kb'])
    if kind == 'potential':
        # a trace keeps the energies in single precision, F(Q)'s own
        e, g = s['pot'].evaluate(s['x'], want_grad=s['gradient'])
        return (e.float(), g) if g is not None else (e.float(),)
    if kind == 'hmc':
        h = s['hmc'].step()
        return h.positions(), h.g
    if kind == 'grad_pdf':
        return debye.grad_pdf(s['grad'], s['qstep'], s['exp']['rstep'],
                              s['rgrid'], s['exp']['qmin'])
    mc = s['mc'].step(s['steps'])
    return mc.positions(), mc.state['accepted'], mc.energies().float()


# ---------------------------------------------------------------- work, exact
def work(case):
    """Every input read and every output written once.  Of the arithmetic
    only what no way of summing avoids is counted: ten operations for the
    distance and the term of each pair."""
    kind = case['kind']
    if kind in ('fq', 'fq_grad', 'grad_fq'):
        n, k = case['n'], GRIDS[case['grid']][1]
        out = (k if kind != 'grad_fq' else 0) + \
            (3 * n * k if kind != 'fq' else 0)
        return {'bytes': 12 * n + 4 * n + 4 * case['species'] * k + 4 * out,
                'flops': 10 * n * (n - 1) / 2}
    if kind == 'batch_fq':
        k = GRIDS[case['grid']][1]
        sizes = np.random.default_rng(case['configs']).integers(
            case['n_min'], case['n_max'] + 1, case['configs'])
        return {'bytes': int(16 * sizes.sum() + 4 * case['species'] * k +
                             4 * k * case['configs']),
                'flops': float((5.0 * sizes * (sizes - 1)).sum())}
    exp, _, k, rgrid = experiment_grids({'rmax': case.get('rmax', 40.0)})
    if kind == 'grad_pdf':
        n = case['n']
        return {'bytes': 12 * n * k + 24 * n * len(rgrid),
                'flops': 2 * 3 * n * k * len(rgrid)}
    n, b = case['n'], case['configs']
    per = 12 * n + 12 * n * bool(case.get('gradient', True)) + 16
    if kind == 'potential':
        return {'bytes': b * per + 8 * len(rgrid),
                'flops': b * (10 * n * (n - 1) / 2 + 2 * k * len(rgrid))}
    if kind == 'hmc':
        return {'bytes': b * per * case['leapfrog'] + 8 * len(rgrid),
                'flops': case['leapfrog'] * b *
                (10 * n * (n - 1) / 2 + 2 * k * len(rgrid))}
    return {'bytes': b * case['steps'] * (24 * k + 12 * n),
            'flops': b * case['steps'] * (20 * n + 2 * k * k)}


@functools.lru_cache(maxsize=4)
def _transform(rmax):
    """F(Q) -> G(r) as a matrix [K, R]: zero pad, odd extension, inverse FFT
    and linear interpolation onto the r grid."""
    exp, qstep, n_bins, rgrid = experiment_grids({'rmax': rmax})
    length = max(n_bins, math.ceil(math.pi / exp['rstep'] / qstep))
    first = int(round(exp['qmin'] / qstep))
    npad = 2 * 2 ** math.ceil(math.log2(first + length))
    x = rgrid / (math.pi / (npad * qstep)) / 2
    lo = x.astype(int)
    w = x - lo
    m = np.arange(n_bins)[:, None]
    ang = 2 * np.pi / npad
    t = (1 - w) * np.sin(ang * ((m * lo) % npad)) + \
        w * np.sin(ang * ((m * (lo + 1)) % npad))
    t *= 2 * qstep / np.pi
    t[:math.ceil(exp['qmin'] / qstep)] = 0
    return t


def _norm(sp, tab):
    """n times the mean of f_i f_j over the pairs, per bin."""
    n = len(sp)
    f = np.asarray(tab, np.float64)
    count = np.bincount(sp, minlength=len(f)).astype(np.float64)
    s1, s2 = count @ f, count @ (f * f)
    return n * ((s1 * s1 - s2) / 2) / (n * (n - 1) / 2)


def _exact_pairs(pos, sp, tab, qbin, kb, grad=False, weights=None,
                 need_f=True):
    """FP64 sums over the pairs of one configuration, bin after bin by the
    three-term recurrence of sin and cos, started anew every 32 bins.
    Returns F(Q) [K], and with ``grad`` the gradient -1/2 dF/dx [N, 3, K] or,
    with ``weights`` [K], sum_k weights_k dF_k/dx [N, 3]."""
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    x = pos.to(device=dev, dtype=torch.float64)
    n = x.shape[0]
    f = torch.as_tensor(np.asarray(tab, np.float64), device=dev)[
        torch.as_tensor(sp, device=dev).long()]                    # [N, K]
    n_bins = f.shape[1]
    na = torch.as_tensor(_norm(sp, tab), device=dev)
    sums = torch.zeros(n_bins, dtype=torch.float64, device=dev)
    want = grad or weights is not None
    out = None
    if want:
        out = torch.zeros((n, 3) if weights is not None else (n, 3, n_bins),
                          dtype=torch.float64, device=dev)
    x4 = torch.cat([x, torch.ones_like(x[:, :1])], 1)
    rows = max(1, min(n, 4_000_000 // n))
    for a in range(0, n, rows):
        xa = x[a:a + rows]
        r2 = ((xa[:, None] - x[None]) ** 2).sum(-1)
        own = torch.arange(xa.shape[0], device=dev)
        r2[own, own + a] = 1.0
        r = r2.sqrt()
        theta = qbin * r
        two_c = 2 * torch.cos(theta)
        ws = 1 / (r2 * r) if want else 1 / r
        ws[own, own + a] = 0
        wc = 1 / r2 if want else None
        if want:
            wc[own, own + a] = 0
        for k in range(max(kb, 0), n_bins):
            if (k - kb) % 32 == 0:
                # t0, t1 (and c0, c1) hold the bins k - 1 and k times their
                # signs g0, g1
                g0 = g1 = 1.0
                t1, t0 = torch.sin(k * theta) * ws, \
                    torch.sin((k - 1) * theta) * ws
                if want:
                    c1, c0 = torch.cos(k * theta) * wc, \
                        torch.cos((k - 1) * theta) * wc
            else:
                t0.addcmul_(two_c, t1, value=-g0 * g1)
                t0, t1 = t1, t0
                if want:
                    c0.addcmul_(two_c, c1, value=-g0 * g1)
                    c0, c1 = c1, c0
                g0, g1 = g1, -g0
            fk = f[:, k]
            if not grad:
                s = t1 @ fk if weights is None else (t1 * r2) @ fk
                sums[k] += g1 * (fk[a:a + rows] @ s) / 2
            elif need_f:
                sums[k] += g1 * (fk[a:a + rows] @ ((t1 * r2) @ fk)) / 2
            if want:
                xf = x4 * fk[:, None]
                m = g1 * (k * qbin * (c1 @ xf) - t1 @ xf)          # [rows, 4]
                row = (-fk[a:a + rows] / na[k])[:, None] * \
                    (xa * m[:, 3:] - m[:, :3])
                if weights is not None:
                    out[a:a + rows] -= 2 * weights[k] * row
                else:
                    out[a:a + rows, :, k] = row.to(out.dtype)
    fq = 2 * sums / na
    fq[:kb] = 0
    return fq, out


def _exact_fq(pos, sp, tab, qbin, kb):
    return _exact_pairs(pos, sp, tab, qbin, kb)[0]


def exact(case, seed):
    kind = case['kind']
    if kind in ('hmc', 'mh'):
        return None     # a chain of random decisions, not a formula
    s = _inputs(case, seed)
    if kind in ('fq', 'fq_grad', 'grad_fq'):
        pos = torch.as_tensor(s['pos'])
        # the gradient costs about ten times F(Q): minutes beyond this size
        grad = kind != 'fq' and case['n'] ** 2 * s['tab'].shape[1] <= 3e10
        if kind == 'grad_fq' and not grad:
            return None
        fq, g = _exact_pairs(pos, s['sp'], s['tab'], s['qbin'], s['kb'],
                             grad=grad, need_f=kind == 'fq_grad')
        return fq if kind == 'fq' else g if kind == 'grad_fq' else (fq, g)
    if kind == 'batch_fq':
        off = s['off']
        return torch.stack([
            _exact_fq(torch.as_tensor(s['pos'][a:b]), s['sp'][a:b], s['tab'],
                      s['qbin'], s['kb']) for a, b in zip(off[:-1], off[1:])])
    if kind == 'grad_pdf':
        g = s['grad'].astype(np.float64)
        return g @ _transform(case['rmax'])
    t = torch.as_tensor(_transform(case['rmax']), device='cuda')
    go = torch.as_tensor(s['gobs'], device='cuda')
    energies, grads = [], []
    for x in s['start']:
        x = torch.as_tensor(x)
        fq = _exact_fq(x, s['sp'], s['tab'], s['qstep'], 0)
        gc = fq @ t
        scale = (gc @ go) / (gc @ gc)
        used = torch.where(scale > 0, scale, torch.ones_like(scale))
        e = go - used * gc
        if case['potential'] == 'rw':
            v = torch.sqrt((e @ e) / (go @ go))
            pre = -v / (e @ e)
        else:
            v, pre = e @ e, -2.0
        energies.append(100.0 * v)
        if case['gradient']:
            c = pre * (used * e + (gc @ e) * (go - 2 * scale * gc) /
                       (gc @ gc))
            grads.append(100.0 * _exact_pairs(
                x, s['sp'], s['tab'], s['qstep'], 0, weights=t @ c)[1])
    energies = torch.stack(energies)
    return (energies, torch.cat(grads)) if grads else (energies,)
