"""GPU parity of the phase-grid kernels (phase_grid.cuh) against the FP64
oracle, at the edges of their tiles, grids and dispatch rules.

Tolerances are the suite's (norm-wise relative): F(Q) and potentials 1e-5,
gradients 1e-4.
"""
import numpy as np
import pytest

from oracle import debye_np as O
from pyiid_gb300.scatter_factors import form_factor_array
from pyiid_gb300 import structures as S

pytestmark = pytest.mark.gpu

TOL_F = 1e-5
TOL_G = 1e-4


def rel(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


@pytest.fixture(scope='module')
def D():
    from pyiid_gb300 import debye
    return debye


def cluster(n, seed, species=1, shift=0.0):
    rng = np.random.default_rng(seed)
    pos = S.displaced(S.fcc_nearest(4.08, n), 0.05, seed) + np.float32(shift)
    nums = rng.choice([46, 78, 79][:species], n) if species > 1 \
        else np.full(n, 79)
    return pos[rng.permutation(n)], nums


def tables(numbers, qb, nb):
    uniq, sp = np.unique(numbers, return_inverse=True)
    tab = np.stack([form_factor_array(z, np.arange(nb) * qb) for z in uniq])
    return sp.reshape(-1).astype(np.int32), tab.astype(np.float32)


# tile edges (31, 32, 33, 65 atoms); one to three elements; a period of Q
# shorter than the cluster (rmax 3: distances beyond half a period fold);
# qmin above some bins; a table too large for shared memory (rmax 110: 887
# bins); a cluster away from the origin; chi^2
@pytest.mark.parametrize('sizes,species,exp,shift,kind', [
    ([31], 1, {}, 0.0, 'rw'),
    ([32], 1, {'rmax': 20.0}, 0.0, 'chi_sq'),
    ([33, 65], 2, {'rmax': 17.3, 'qmin': 0.9}, 0.0, 'rw'),
    ([97], 3, {'rmax': 3.0}, 0.0, 'rw'),
    ([64], 2, {'rmax': 110.0, 'rstep': 0.05}, 0.0, 'rw'),
    ([120], 1, {'rmax': 12.0, 'qmax': 7.0}, 150.0, 'rw'),
    ([300, 1, 0, 280], 2, {'rmax': 20.0}, -60.0, 'chi_sq'),
])
def test_pair_force_table_matches_oracle(D, sizes, species, exp, shift, kind):
    import torch
    e = O.update_experiment(dict({'rstep': 0.02}, **exp))
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    parts = [cluster(n, 7 + n, species, shift) for n in sizes]
    pos = np.concatenate([p for p, _ in parts]).astype(np.float32)
    sp, tab = tables(np.concatenate([z for _, z in parts]), qb, nb)
    off = np.concatenate([[0], np.cumsum(sizes)])
    ref = S.fcc_nearest(4.0, 50).astype(np.float32)
    gobs = O.pdf_fft(O.fq(ref, np.repeat(tab[:1], 50, 0), qb), e['rstep'], qb,
                     rg, e['qmin'])
    out = D.batch_potential_grad(pos, sp, off, tab, qb, e['rstep'], rg,
                                 e['qmin'], torch.as_tensor(gobs), kind)
    g = out['grad'].cpu().numpy()
    for i, n in enumerate(sizes):
        if n < 2:
            continue
        a, b = off[i], off[i + 1]
        val, tg = O.true_grad_potential(pos[a:b], tab[sp[a:b]], e, gobs, kind)
        assert abs(out['energy'][i, 0].item() - val) <= TOL_F * abs(val)
        assert rel(g[a:b], tg) <= TOL_G, (i, rel(g[a:b], tg))


# The length of an item's run of tiles grows with the tile pairs of the call
# (about four items per SM: one tile up to 1,215 pairs; here also two, three,
# five and nine), and with it how the warps share its steps and where the
# table is read.  Copies of one configuration need one oracle evaluation.
@pytest.mark.parametrize('n,species,copies,exp', [
    (165, 1, 40, {}),
    (165, 1, 64, {}),
    (240, 2, 40, {}),
    (193, 1, 70, {}),
    (290, 2, 64, {}),
    (290, 1, 100, {}),
    (290, 1, 64, {'rmax': 110.0, 'rstep': 0.05}),
])
def test_pair_force_of_longer_runs_matches_oracle(D, n, species, copies, exp):
    import torch
    e = O.update_experiment(dict({'rstep': 0.02, 'rmax': 40.0}, **exp))
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    pos, nums = cluster(n, 11 + n, species)
    sp, tab = tables(nums, qb, nb)
    gobs = O.pdf_fft(O.fq(S.fcc_nearest(4.0, 50), np.repeat(tab[:1], 50, 0),
                          qb), e['rstep'], qb, rg, e['qmin'])
    out = D.batch_potential_grad(
        np.tile(pos, (copies, 1)), np.tile(sp, copies),
        np.arange(copies + 1) * n, tab, qb, e['rstep'], rg, e['qmin'],
        torch.as_tensor(gobs))
    g = out['grad'].cpu().numpy().reshape(copies, n, 3)
    val, tg = O.true_grad_potential(pos, tab[sp], e, gobs)
    energy = out['energy'][:, 0].cpu().numpy()
    assert np.all(np.abs(energy - val) <= TOL_F * abs(val))
    for i in range(copies):
        assert rel(g[i], tg) <= TOL_G, (i, rel(g[i], tg))


def test_pair_force_table_close_and_coincident_pairs(D):
    """Pairs nearer than the split coordinates resolve (0.1 A) take the
    general distance; coincident atoms give NaN rows, the others' stay."""
    import torch
    e = O.update_experiment({'rmax': 20.0, 'rstep': 0.02})
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    pos, nums = cluster(80, 5)
    pos[11] = pos[40] + np.float32([0.03, -0.02, 0.01])
    sp, tab = tables(nums, qb, nb)
    gobs = O.pdf_fft(O.fq(S.fcc_nearest(4.0, 50), np.repeat(tab, 50, 0), qb),
                     e['rstep'], qb, rg, e['qmin'])
    args = (sp, np.array([0, 80]), tab, qb, e['rstep'], rg, e['qmin'],
            torch.as_tensor(gobs))
    g = D.batch_potential_grad(pos, *args)['grad'].cpu().numpy()
    _, tg = O.true_grad_potential(pos, tab[sp], e, gobs)
    assert rel(g, tg) <= TOL_G
    pos[11] = pos[40]
    g = D.batch_potential_grad(pos, *args)['grad'].cpu().numpy()
    assert np.all(np.isnan(g[[11, 40]]))


def fq64(pos, sp, tab, qb):
    return O.fq(np.asarray(pos, np.float32), tab[sp], qb)


# sizes either side of the rule that takes a call to the grid; odd bin counts
# (M is rounded up to a multiple of 4); two and three elements; k_begin odd;
# a period shorter than the cluster; a cluster away from the origin
@pytest.mark.parametrize('n,species,qb,nb,kb,shift', [
    (380, 1, 0.05, 500, 2, 0.0),
    (421, 1, 0.05, 501, 3, 25.0),
    (600, 2, 0.05, 499, 0, 0.0),
    (260, 1, 0.02, 1475, 25, -70.0),
    (700, 1, 0.4, 250, 1, 0.0),
    (640, 3, 0.02, 1502, 0, 0.0),
])
def test_fq_on_the_grid_matches_oracle(D, n, species, qb, nb, kb, shift):
    pos, nums = cluster(n, n, species, shift)
    sp, tab = tables(nums, qb, nb)
    f = D.fq(pos, sp, tab, qb, k_begin=kb).cpu().numpy()
    f2 = D.fq(pos, sp, tab, qb, k_begin=kb).cpu().numpy()
    assert np.array_equal(f, f2) and np.all(f[:kb] == 0)
    idx = np.unique(np.concatenate([np.arange(kb, nb, 7), [nb - 1]]))
    x = pos.astype(np.float64)
    fi = tab[sp][:, idx].astype(np.float64)
    s = np.zeros(len(idx))
    for a in range(1, n):
        d = np.sqrt(((x[a] - x[:a]) ** 2).sum(1))[:, None]
        s += fi[a] * (fi[:a] * np.sin(idx * qb * d) / d).sum(0)
    want = 2 * s / O.normalization(tab[sp])[idx]
    assert rel(f[idx], want) <= TOL_F, rel(f[idx], want)


def test_fq_on_the_grid_close_coincident_and_far_pairs(D):
    """Pairs at tiny distances (power sums), under 0.1 A and beyond 128 A
    (general distance) against the oracle; a coincident pair makes every bin
    0, as the reference's NaN does, and so does a NaN position, in its own
    configuration only."""
    qb, nb = 0.05, 300
    pos, nums = cluster(420, 9, 2)
    pos[30] = pos[7] + np.float32([1e-3, 0, 0])
    pos[31] = pos[8] + np.float32([0.02, 0.03, 0.01])
    pos[32] += np.float32([150.0, 0, 0])
    sp, tab = tables(nums, qb, nb)
    want = fq64(pos, sp, tab, qb)
    assert rel(D.fq(pos, sp, tab, qb).cpu().numpy(), want) <= TOL_F
    bad = pos.copy()
    bad[30] = bad[7]
    nan = pos.copy()
    nan[5, 1] = np.nan
    both = np.concatenate([bad, pos, nan])
    f = D.batch_fq(both, np.tile(sp, 3), np.array([0, 420, 840, 1260]), tab,
                   qb).cpu().numpy()
    assert np.all(f[0] == 0) and np.all(f[2] == 0)
    assert rel(f[1], want) <= TOL_F


def test_mixed_batch_of_grid_and_direct_configurations(D):
    """Small configurations of a batch stay on the direct kernels beside the
    ones on the grid; a CUDA graph replay equals the eager call bitwise."""
    import torch
    qb, nb = 0.05, 500
    sizes = [3, 500, 0, 60, 450, 1, 33, 600]
    parts = [cluster(n, 60 + n, 2) for n in sizes if n]
    pos = torch.as_tensor(np.concatenate([p for p, _ in parts]).astype(
        np.float32), device='cuda')
    sp, tab = tables(np.concatenate([z for _, z in parts]), qb, nb)
    off = np.concatenate([[0], np.cumsum(sizes)])
    f = D.batch_fq(pos, sp, off, tab, qb, 2)
    out = torch.empty_like(f)
    D.batch_fq(pos, sp, off, tab, qb, 2, out=out)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        D.batch_fq(pos, sp, off, tab, qb, 2, out=out)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, f)
    p = pos.cpu().numpy()
    for i, n in enumerate(sizes):
        a, b = off[i], off[i + 1]
        got = f[i].cpu().numpy()
        if n < 2:
            assert np.all(got == 0)
        else:
            assert rel(got[2:], fq64(p[a:b], sp[a:b], tab, qb)[2:]) <= TOL_F


# tile and column edges (31 to 97 atoms); one to three elements; a period of Q
# far shorter than the cluster (q step 0.7: pairs several periods apart, the
# second sweep); the shortest and longest transforms and the first bin count
# beyond them (2,008, the direct kernels); odd and zero k_begin; one bin
# above k_begin; a cluster away from the origin
@pytest.mark.parametrize('n,species,qb,nb,kb,shift', [
    (32, 1, 0.05, 500, 2, 0.0),
    (33, 1, 0.1, 187, 1, 30.0),
    (65, 2, 0.1, 250, 0, 0.0),
    (97, 3, 0.05, 301, 3, -200.0),
    (64, 1, 0.7, 90, 0, 0.0),
    (97, 2, 0.45, 250, 5, 0.0),
    (40, 1, 0.012, 2007, 25, 0.0),
    (40, 1, 0.012, 2008, 25, 0.0),
    (64, 1, 0.05, 400, 399, 0.0),
    (64, 1, 0.02, 1475, 25, 0.0),
])
def test_gradient_on_the_grid_matches_oracle(D, n, species, qb, nb, kb, shift):
    pos, nums = cluster(n, n, species, shift)
    sp, tab = tables(nums, qb, nb)
    f, g = (t.cpu().numpy() for t in D.fq_grad(pos, sp, tab, qb, k_begin=kb))
    g1 = D.grad_fq(pos, sp, tab, qb, k_begin=kb).cpu().numpy()
    want_f = fq64(pos, sp, tab, qb)
    want_g = O.grad_fq(pos, tab[sp], qb)
    assert np.all(f[:kb] == 0)
    assert np.all(g[:, :, :kb] == 0) and np.all(g1[:, :, :kb] == 0)
    assert rel(f[kb:], want_f[kb:]) <= TOL_F
    assert rel(g[:, :, kb:], want_g[:, :, kb:]) <= TOL_G
    assert rel(g1[:, :, kb:], want_g[:, :, kb:]) <= TOL_G


def test_gradient_on_the_grid_close_coincident_and_far_pairs(D):
    """Pairs at tiny distances, under 0.1 A, beyond 128 A and several periods
    apart, each against the oracle's rows; the rows of a coincident pair are
    0 and F is 0, the others' rows stay."""
    qb, nb = 0.3, 250
    pos, nums = cluster(90, 19, 2)
    pos[30] = pos[7] + np.float32([2e-4, 1e-4, 0])
    pos[31] = pos[8] + np.float32([0.02, 0.03, 0.01])
    pos[32] += np.float32([150.0, 0, 0])
    sp, tab = tables(nums, qb, nb)
    f, g = (t.cpu().numpy() for t in D.fq_grad(pos, sp, tab, qb))
    want = O.grad_fq(pos, tab[sp], qb)
    assert rel(f, fq64(pos, sp, tab, qb)) <= TOL_F
    for a in (7, 30, 8, 31, 32, 50):
        assert rel(g[a], want[a]) <= TOL_G, (a, rel(g[a], want[a]))
    bad = pos.copy()
    bad[30] = bad[7]
    f, g = (t.cpu().numpy() for t in D.fq_grad(bad, sp, tab, qb))
    assert np.all(f == 0) and np.all(g[[7, 30]] == 0)
    want = O.grad_fq(bad, tab[sp], qb)
    keep = np.setdiff1d(np.arange(90), [7, 30])
    assert rel(g[keep], want[keep]) <= TOL_G


def test_gradient_on_the_grid_under_capture(D):
    """One element with more columns than warps, and three whose blocks end
    inside a CTA's share of the columns: eager, repeated and graph-replayed
    calls are bitwise equal, also into an output at an odd offset."""
    import torch
    for n, species in ((400, 1), (460, 3)):
        pos, nums = cluster(n, n, species)
        sp, tab = tables(nums, 0.05, 300)
        p = torch.as_tensor(pos.astype(np.float32), device='cuda')
        f, g = D.fq_grad(p, sp, tab, 0.05, 1)
        big = torch.full((n * 900 + 4,), float('nan'), device='cuda')
        out = big[1:1 + n * 900].view(n, 3, 300)
        f2 = torch.empty_like(f)
        D.fq_grad(p, sp, tab, 0.05, 1, out_fq=f2, out_grad=out)
        assert torch.equal(f2, f) and torch.equal(out, g)
        assert torch.isnan(big[0]) and torch.isnan(big[-3:]).all()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            D.fq_grad(p, sp, tab, 0.05, 1, out_fq=f2, out_grad=out)
        out.zero_()
        f2.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(f2, f) and torch.equal(out, g)
        assert rel(f.cpu().numpy()[1:], fq64(pos, sp, tab, 0.05)[1:]) <= TOL_F


# one, two and eight CTAs per cluster (100, 60, 3 configurations), eight
# configurations at a time with a remainder, bins in part of a block, qmin
# above the first block, few and odd points
@pytest.mark.parametrize('n_configs,exp', [
    (1, {'rmax': 20.0}), (3, {'rmax': 7.01, 'rstep': 0.03}),
    (8, {'rmax': 33.0, 'qmin': 3.3}), (60, {'rmax': 20.0, 'qmin': 0.5}),
    (101, {'rmax': 12.0, 'rstep': 0.05}),
])
def test_transform_and_potential_of_batches(D, n_configs, exp):
    import torch
    e = O.update_experiment(dict({'rstep': 0.02}, **exp))
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    rng = np.random.default_rng(n_configs)
    fq = rng.normal(0, 1, (n_configs, nb)).astype(np.float32)
    gr = D.pdf(torch.as_tensor(fq, device='cuda'), qb, e['rstep'], rg,
               e['qmin'])
    want = np.stack([O.pdf_fft(f.astype(np.float64), e['rstep'], qb, rg,
                               e['qmin']) for f in fq])
    assert rel(gr.cpu().numpy(), want) <= TOL_F
    gobs = want[0] + rng.normal(0, .3, len(rg))
    g = torch.as_tensor(want, device='cuda')
    w = torch.as_tensor(rng.random(len(rg)), device='cuda')
    for kind, f in (('rw', O.get_rw), ('chi_sq', O.get_chi_sq)):
        got = D.potential(torch.as_tensor(gobs), g, kind).cpu().numpy()
        for i in range(n_configs):
            v, s = f(gobs, want[i])
            assert abs(got[i, 0] - v) <= 1e-12 * abs(v)
            assert abs(got[i, 1] - s) <= 1e-12 * abs(s)
    got = D.potential(torch.as_tensor(gobs), g, 'rw', weight=w).cpu().numpy()
    wn = w.cpu().numpy()
    for i in range(n_configs):
        a = (want[i] @ gobs) / (want[i] @ want[i])
        v = 1.0 if a <= 0 else np.sqrt((wn * (gobs - a * want[i]) ** 2).sum() /
                                       (wn * gobs ** 2).sum())
        assert abs(got[i, 0] - v) <= 1e-12 * abs(v)


def sampled_fq(pos, sp, tab, qb, bins):
    """F on `bins` from FP64 pair sums."""
    from oracle import debye_c as C
    bins = np.asarray(bins, np.int32)
    return 2 * C.pair_sums(pos, sp, tab, qb, bins) / \
        O.normalization(tab[sp])[bins]


# A warp's share of a key's columns grows with the batch: thousands of values
# per copy of a cell here.  Their error must not: the bound
# is twice what the direct kernels, which add short FP32 sums in FP64, leave
# for one such particle (2e-7); sums held in FP32 alone leave 1.2e-6.
def test_sums_of_a_large_batch_keep_their_precision(D):
    n, copies, qb, nb = 20000, 16, 0.02, 1500
    pos, nums = cluster(n, 3)
    sp, tab = tables(nums, qb, nb)
    f = D.batch_fq(np.tile(pos, (copies, 1)), np.tile(sp, copies),
                   np.arange(copies + 1) * n, tab, qb).cpu().numpy()
    bins = np.arange(41, nb, 97)
    want = sampled_fq(pos, sp, tab, qb, bins)
    for row in f:
        assert rel(row[bins], want) <= 4e-7, rel(row[bins], want)


# The transform of many pairs at the bins where FP32 rotations would see the
# small-angle peak of F (multiples of M / 33 of M = 5 n_bins cells).  Bound:
# the rounding of the sums handed to it (4e-8), the window (2e-8) and the
# distances (5e-8), added and rounded up.
@pytest.mark.parametrize('grad', [False, True])
def test_transform_of_a_large_particle(D, grad):
    n, qb, nb = 30000, 0.02, 1500
    pos, nums = cluster(n, 4)
    sp, tab = tables(nums, qb, nb)
    m = 6144 if grad else 5 * nb
    bins = np.round(m / 33 * np.arange(1, 6)).astype(int)
    f = D.fq_grad(pos, sp, tab, qb)[0] if grad else D.fq(pos, sp, tab, qb)
    want = sampled_fq(pos, sp, tab, qb, bins)
    assert rel(f.cpu().numpy()[bins], want) <= 1.5e-7, \
        rel(f.cpu().numpy()[bins], want)


# Most pairs beyond 128 A, where the split coordinates no longer give the
# distance: a rod, and two clusters far apart.
@pytest.mark.parametrize('shape', ['rod', 'halves'])
def test_far_pairs_match_oracle(D, shape):
    from oracle import debye_c as C
    n, qb, nb, kb = 700, 0.05, 500, 2
    if shape == 'rod':
        pos = np.zeros((n, 3), np.float32)
        pos[:, 0] = 2.9 * np.arange(n)
        pos += np.random.default_rng(6).normal(0, 0.05, pos.shape)
        pos = pos.astype(np.float32)
        nums = np.full(n, 79)
    else:
        pos, nums = cluster(n, 8, 2)
        pos[::2] += np.float32([300.0, -250.0, 100.0])
    sp, tab = tables(nums, qb, nb)
    bins = np.arange(kb, nb, 11)
    want = sampled_fq(pos, sp, tab, qb, bins)
    f = D.fq(pos, sp, tab, qb, kb).cpu().numpy()
    f2, g = (t.cpu().numpy() for t in D.fq_grad(pos, sp, tab, qb, kb))
    assert rel(f[bins], want) <= TOL_F and rel(f2[bins], want) <= TOL_F
    rows = np.array([0, 1, n // 2, n - 1], np.int32)
    want_g = -C.grad_rows(pos, sp, tab, qb, rows) / O.normalization(tab[sp])
    for i, a in enumerate(rows):
        assert rel(g[a, :, kb:], want_g[i, :, kb:]) <= TOL_G


# ... which are no rare case to be done one at a time: the same two clusters
# 400 A apart instead of 100 take about one distance in full more per pair,
# not twice as long.
def test_far_pairs_cost_what_near_ones_cost(D):
    import torch
    n, qb, nb = 4000, 0.05, 500
    pos, nums = cluster(n, 12)
    sp, tab = tables(nums, qb, nb)

    def ms(fn):
        fn()
        t = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(4):
                fn()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return np.median(t)

    def times(apart):
        p = pos.copy()
        p[::2, 0] += np.float32(apart)
        p = torch.as_tensor(p, device='cuda')
        return (ms(lambda: D.fq(p, sp, tab, qb)),
                ms(lambda: D.fq_grad(p, sp, tab, qb)))

    near, far = times(100.0), times(400.0)
    assert far[0] <= 2 * near[0] and far[1] <= 2 * near[1], (near, far)
