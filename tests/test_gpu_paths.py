"""Which kernels a call runs, and parity of the direct pair kernels (those
with launch variants) at sizes that the dispatch rules leave to them.

Each test states the path it is about through Context.variant_launches, so a
rule that moves its sizes elsewhere makes it fail instead of emptying it.
Tolerances as everywhere (norm-wise relative): F(Q) and potentials 1e-5,
gradients 1e-4.
"""
import numpy as np
import pytest

from oracle import debye_c as C
from oracle import debye_np as O
from pyiid_gb300 import structures as S
from pyiid_gb300.scatter_factors import form_factor_array, species_tables

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


@pytest.fixture
def ctx():
    """The shared context, its variants as they were afterwards."""
    from pyiid_gb300 import autotune
    with autotune.variant_scope() as c:
        yield c


def launched(ctx, kernel, fn):
    """(launches of ``kernel``'s variants, result) of one call."""
    n = ctx.variant_launches(kernel)
    out = fn()
    return ctx.variant_launches(kernel) - n, out


def particle(n, seed, species=1):
    rng = np.random.default_rng(seed)
    pos = S.displaced(S.fcc_nearest(4.08, n), 0.05, seed)[rng.permutation(n)]
    nums = rng.choice([46, 78, 79][:species], n) if species > 1 \
        else np.full(n, 79)
    return pos.astype(np.float32), nums


def fq64(pos, sp, tab, qb, bins):
    bins = np.asarray(bins, np.int32)
    return 2 * C.pair_sums(pos, sp, tab, qb, bins) / \
        O.normalization(tab[sp])[bins]


def rows64(pos, sp, tab, qb, rows):
    return -C.grad_rows(pos, sp, tab, qb, np.asarray(rows, np.int32)) / \
        O.normalization(tab[sp])


# fewer than 64 bins, and more than the grid has: several tiles per work item
# (1,300 atoms), one element and two
@pytest.mark.parametrize('n,species,nb', [(70, 2, 500), (1300, 1, 60),
                                          (1300, 2, 60), (300, 2, 2900)])
def test_direct_fq_variants_match_oracle(D, ctx, n, species, nb):
    from pyiid_gb300 import autotune
    pos, nums = particle(n, n, species)
    qb, kb = 0.02 if nb > 500 else 0.1, 3
    sp, tab, _ = species_tables(nums, qb, nb)
    bins = np.unique(np.concatenate([np.arange(kb, nb, nb // 40 + 1),
                                     [nb - 1]]))
    want = fq64(pos, sp, tab, qb, bins)
    for idx, info in autotune.variants('fq'):
        ctx.set_variant('fq', idx)
        ran, f = launched(ctx, 'fq', lambda: D.fq(pos, sp, tab, qb, kb))
        f = f.cpu().numpy()
        assert ran == 1
        assert np.all(f[:kb] == 0)
        assert rel(f[bins], want) <= TOL_F, (idx, info)


def test_direct_persistent_batch_equals_one_cta_per_unit(D, ctx):
    from pyiid_gb300 import autotune
    rng = np.random.default_rng(31)
    sizes = [int(n) for n in rng.integers(2, 90, 40)]
    parts = [particle(n, 80 + i, 2) for i, n in enumerate(sizes)]
    pos = np.concatenate([p for p, _ in parts])
    off = np.concatenate([[0], np.cumsum(sizes)])
    sp, tab, _ = species_tables(np.concatenate([z for _, z in parts]), 0.05,
                                500)
    shapes = {(i['bins_per_thread'], i['pairs_per_thread']): idx
              for idx, i in autotune.variants('fq')}
    got = {}
    for shape in ((56, -3), (56, -13), (56, -13)):
        ctx.set_variant('fq', shapes[shape])
        ran, f = launched(ctx, 'fq', lambda: D.batch_fq(pos, sp, off, tab,
                                                        0.05, 2))
        assert ran == 1
        assert np.array_equal(got.setdefault('f', f.cpu().numpy()),
                              f.cpu().numpy())
    for i in (0, 7, 39):
        a, b = off[i], off[i + 1]
        assert rel(got['f'][i, 2:], O.fq(pos[a:b], tab[sp[a:b]], 0.05)[2:]) \
            <= TOL_F


# beyond the longest transform (2,007 bins); 33 and 70 atoms of two elements
# (tile remainders), 300 of three (tiles J split over CTAs)
@pytest.mark.parametrize('n,species', [(33, 2), (70, 2), (300, 3)])
@pytest.mark.parametrize('kernel', ['grad_fq', 'fq_grad'])
def test_direct_gradient_variants_match_oracle(D, ctx, kernel, n, species):
    from pyiid_gb300 import autotune
    pos, nums = particle(n, 2 * n, species)
    qb, nb, kb = 0.012, 2101, 3
    sp, tab, _ = species_tables(nums, qb, nb)
    rows = [0, n // 3, n - 1]
    want_g = rows64(pos, sp, tab, qb, rows)[:, :, kb:]
    bins = np.arange(kb, nb, 53)
    want_f = fq64(pos, sp, tab, qb, bins)
    for idx, info in autotune.variants(kernel):
        ctx.set_variant(kernel, idx)
        if kernel == 'grad_fq':
            ran, g = launched(ctx, kernel,
                              lambda: D.grad_fq(pos, sp, tab, qb, kb))
        else:
            ran, (f, g) = launched(ctx, kernel,
                                   lambda: D.fq_grad(pos, sp, tab, qb, kb))
            f = f.cpu().numpy()
            assert np.all(f[:kb] == 0)
            assert rel(f[bins], want_f) <= TOL_F, (idx, info)
        assert ran == 1
        g = g.cpu().numpy()
        assert np.all(g[:, :, :kb] == 0)
        assert rel(g[rows][:, :, kb:], want_g) <= TOL_G, (idx, info)


def test_direct_split_combine_into_an_output_at_an_odd_offset(D, ctx):
    """A J-split gradient (coefficients, parts, their combination and F) into
    an output 4 bytes past a 16-byte boundary equals the aligned call."""
    import torch
    n, qb, nb, kb = 100, 0.012, 2101, 2
    pos, nums = particle(n, 3)
    sp, tab, _ = species_tables(nums, qb, nb)
    before = ctx.launches
    ran, (f, g) = launched(ctx, 'fq_grad',
                           lambda: D.fq_grad(pos, sp, tab, qb, kb))
    assert ran == 1 and ctx.launches - before == 4  # 3 without a split
    big = torch.full((n * 3 * nb + 4,), float('nan'), device='cuda')
    out = big[1:1 + n * 3 * nb].view(n, 3, nb)
    assert out.data_ptr() % 16 == 4
    f2, g2 = D.fq_grad(pos, sp, tab, qb, kb, out_grad=out)
    assert torch.equal(g2, g) and torch.equal(f2, f)
    assert torch.isnan(big[0]) and torch.isnan(big[-3:]).all()


# few pairs for many (configuration, species pair) tables: one element in
# single and several tiles, two elements; both forms of the kernel
@pytest.mark.parametrize('variant', [0, 1])
@pytest.mark.parametrize('sizes,species,exp', [
    ([70, 33, 97, 5, 64, 80, 31, 32, 96, 40, 75, 66], 1, {'rmax': 40.0}),
    ([70, 33, 97], 2, {'rmax': 60.0}),
    ([130] * 24, 2, {'rmax': 20.0, 'qmin': 0.9}),
])
def test_direct_adjoint_variants_match_oracle(D, ctx, sizes, species, exp,
                                              variant):
    import torch
    e = O.update_experiment(dict({'rstep': 0.02, 'rmax': 30.0}, **exp))
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    parts = [particle(n, 200 + i, species) for i, n in enumerate(sizes)]
    pos = np.concatenate([p for p, _ in parts])
    nums = np.concatenate([z for _, z in parts])
    off = np.concatenate([[0], np.cumsum(sizes)])
    uniq, sp = np.unique(nums, return_inverse=True)
    sp = sp.reshape(-1).astype(np.int32)
    tab = np.stack([form_factor_array(z, np.arange(nb) * qb)
                    for z in uniq]).astype(np.float32)
    gobs = O.pdf_fft(O.fq(S.random_cube(50, 9.0, 3), np.repeat(tab[:1], 50, 0),
                          qb), e['rstep'], qb, rg, e['qmin'])
    ctx.set_variant('adjoint', variant)
    ran, out = launched(ctx, 'adjoint', lambda: D.batch_potential_grad(
        pos, sp, off, tab, qb, e['rstep'], rg, e['qmin'],
        torch.as_tensor(gobs)))
    assert ran == 1
    g = out['grad'].cpu().numpy()
    for i in range(min(3, len(sizes))):
        a, b = off[i], off[i + 1]
        _, tg = O.true_grad_potential(pos[a:b], tab[sp[a:b]], e, gobs)
        assert rel(g[a:b], tg) <= TOL_G, (variant, i, rel(g[a:b], tg))


# either side of the rules, far from the line
@pytest.mark.parametrize('n,species,nb,kb,direct', [
    (55, 1, 250, 0, True), (250, 2, 500, 2, True), (700, 1, 500, 2, False),
    (900, 2, 500, 2, False), (2000, 1, 63, 0, True),
])
def test_fq_path(D, ctx, n, species, nb, kb, direct):
    pos, nums = particle(n, n, species)
    sp, tab, _ = species_tables(nums, 0.05, nb)
    ran, _ = launched(ctx, 'fq', lambda: D.fq(pos, sp, tab, 0.05, kb))
    assert ran == direct


# the direct kernels skip the bins below k_begin, the grid does not: (two
# elements) the same call for all bins and for the last few
@pytest.mark.parametrize('n,copies,nb,kb', [(160, 64, 500, 450),
                                            (200, 64, 1500, 1490),
                                            (300, 1, 2500, 2450)])
def test_fq_path_of_the_last_bins(D, ctx, n, copies, nb, kb):
    pos, nums = particle(n, n, 2)
    sp, tab, _ = species_tables(nums, 0.02, nb)
    pos, sp = np.tile(pos, (copies, 1)), np.tile(sp, copies)
    off = np.arange(copies + 1) * n
    all_bins = launched(ctx, 'fq',
                        lambda: D.batch_fq(pos, sp, off, tab, 0.02))
    last = launched(ctx, 'fq',
                    lambda: D.batch_fq(pos, sp, off, tab, 0.02, kb))
    assert all_bins[0] == 0 and last[0] == 1
    f, g = all_bins[1].cpu().numpy(), last[1].cpu().numpy()
    assert np.all(g[:, :kb] == 0)
    assert rel(g[:, kb:], f[:, kb:]) <= TOL_F


@pytest.mark.parametrize('kernel', ['grad_fq', 'fq_grad'])
def test_gradient_path_of_the_last_bins(D, ctx, kernel):
    n, nb, kb = 900, 1500, 1470
    pos, nums = particle(n, n, 3)
    sp, tab, _ = species_tables(nums, 0.02, nb)
    call = getattr(D, kernel)
    all_bins = launched(ctx, kernel, lambda: call(pos, sp, tab, 0.02))
    last = launched(ctx, kernel, lambda: call(pos, sp, tab, 0.02, kb))
    assert all_bins[0] == 0 and last[0] == 1
    g, g1 = ((x[1] if kernel == 'fq_grad' else x).cpu().numpy()
             for x in (all_bins[1], last[1]))
    assert np.all(g1[:, :, :kb] == 0)
    assert rel(g1[:, :, kb:], g[:, :, kb:]) <= TOL_G


def test_grid_fq_close_coincident_and_far_pairs(D, ctx):
    """Pairs at tiny distances (power sums), under 0.1 A and beyond 128 A
    (general distance) against the oracle; a coincident pair makes every bin
    0, and so does a NaN position, in its own configuration only."""
    qb, nb, n = 0.05, 500, 700
    pos, nums = particle(n, 9, 2)
    pos[30] = pos[7] + np.float32([1e-3, 0, 0])
    pos[31] = pos[8] + np.float32([0.02, 0.03, 0.01])
    pos[32] += np.float32([150.0, 0, 0])
    sp, tab, _ = species_tables(nums, qb, nb)
    bins = np.arange(0, nb, 9)
    want = fq64(pos, sp, tab, qb, bins)
    ran, f = launched(ctx, 'fq', lambda: D.fq(pos, sp, tab, qb))
    assert ran == 0 and rel(f.cpu().numpy()[bins], want) <= TOL_F
    bad, nan, inf = pos.copy(), pos.copy(), pos.copy()
    bad[30] = bad[7]
    nan[5, 1] = np.nan
    inf[6, 2] = np.inf
    ran, f = launched(ctx, 'fq', lambda: D.batch_fq(
        np.concatenate([bad, pos, nan, pos, inf]), np.tile(sp, 5),
        np.arange(6) * n, tab, qb))
    f = f.cpu().numpy()
    assert ran == 0 and np.all(f[[0, 2, 4]] == 0)
    assert rel(f[1, bins], want) <= TOL_F and rel(f[3, bins], want) <= TOL_F


# A gradient whose rows exceed the workspace limit runs in parts of its atoms:
# parts of many and of one or two atoms, parts that begin inside a species and
# at its edge, a species of the table without atoms, a period of Q shorter than
# the cluster (the second rows).  F and dF/dx against one part (the sums are
# cut differently: FP32 roundings) and against the oracle.
@pytest.mark.parametrize('n,species,nb,qb,at_once', [
    (300, 1, 500, 0.05, 100), (301, 2, 500, 0.05, 64), (420, 3, 301, 0.05, 17),
    (48, 1, 500, 0.05, 1), (90, 2, 250, 0.45, 30),
])
def test_gradient_in_parts(D, ctx, n, species, nb, qb, at_once):
    pos, nums = particle(n, n, species)
    sp, tab, _ = species_tables(nums, qb, nb)
    if species != 2:  # a species of the table has no atoms
        sp = np.where(sp > 0, sp + 1, 0).astype(np.int32)
        tab = np.insert(tab, 1, tab[0], axis=0)
    kb = 2
    half = next(x for x in (384, 512, 768, 1024) if 2 * x >= 4.08 * nb)
    row = 24 * (half + 16)
    rows = np.array([0, 1, n // 2, n - 1])
    want_g = rows64(pos, sp, tab, qb, rows)
    f, g = D.fq_grad(pos, sp, tab, qb, kb)
    want_f = fq64(pos, sp, tab, qb, np.arange(kb, nb))
    try:
        # (rows of the warps besides; half a row against the rounding)
        ctx.set_workspace_limit(int((16 * 152 + species * at_once + .5) * row))
        before = ctx.launches
        ran, (f2, g2) = launched(ctx, 'fq_grad',
                                 lambda: D.fq_grad(pos, sp, tab, qb, kb))
        assert ran == 0
        assert ctx.launches - before == 2 + 2 * -(-n // at_once)
        ran, g3 = launched(ctx, 'grad_fq',
                           lambda: D.grad_fq(pos, sp, tab, qb, kb))
        assert ran == 0
        ctx.set_workspace_limit(0)
        ran, (f4, g4) = launched(ctx, 'fq_grad',
                                 lambda: D.fq_grad(pos, sp, tab, qb, kb))
        assert ran == 1
    finally:
        ctx.set_workspace_limit(2 << 30)
    for h in (f, f2, f4):
        h = h.cpu().numpy()
        assert np.all(h[:kb] == 0) and rel(h[kb:], want_f) <= TOL_F
    assert rel(f2.cpu().numpy(), f.cpu().numpy()) <= 1e-6
    for h in (g, g2, g3, g4):
        h = h.cpu().numpy()
        assert np.all(h[:, :, :kb] == 0)
        assert rel(h[rows][:, :, kb:], want_g[:, :, kb:]) <= TOL_G
    assert rel(g2.cpu().numpy(), g.cpu().numpy()) <= 1e-6
    assert rel(g3.cpu().numpy(), g.cpu().numpy()) <= 1e-6


def test_default_workspace_limit_bounds_a_large_gradient(D, ctx):
    """7,000 atoms of three elements at 2,007 bins would need 2.3 GB of rows:
    two parts within 2 GiB, sampled rows and bins against FP64."""
    import torch
    n, qb, nb, kb = 7000, 0.015, 2007, 3
    pos, nums = particle(n, 7, 3)
    sp, tab, _ = species_tables(nums, qb, nb)
    before = ctx.launches
    ran, (f, g) = launched(ctx, 'fq_grad',
                           lambda: D.fq_grad(pos, sp, tab, qb, kb))
    assert ran == 0 and ctx.launches - before == 2 + 2 * 2
    bins = np.arange(kb, nb, 127)
    assert rel(f.cpu().numpy()[bins], fq64(pos, sp, tab, qb, bins)) <= TOL_F
    rows = np.array([0, 3499, 3500, n - 1])
    want = rows64(pos, sp, tab, qb, rows)
    got = g[torch.as_tensor(rows, device=g.device)].cpu().numpy()
    for i in range(len(rows)):
        assert rel(got[i, :, kb:], want[i, :, kb:]) <= TOL_G


def test_many_ranges_of_bins_allocate_nothing_once_warm(D, ctx):
    """A batch of grid and direct configurations and a gradient, each at 20
    bin counts: warm calls make no allocation (all are captured in one graph),
    and a replay equals the eager calls."""
    import torch
    sizes = [500, 3, 60, 450, 800]
    parts = [particle(n, 60 + n, 2) for n in sizes]
    pos = torch.as_tensor(np.concatenate([p for p, _ in parts]), device='cuda')
    off = np.concatenate([[0], np.cumsum(sizes)])
    _, sp = np.unique(np.concatenate([z for _, z in parts]),
                      return_inverse=True)
    sp = sp.reshape(-1).astype(np.int32)
    counts = list(range(400, 420))
    # (a context holds one form-factor table, so all of these are alike)
    tabs = {nb: np.full((2, nb), 2.0, np.float32) for nb in counts}
    n1 = sizes[0]

    def calls(out):
        for nb in counts:
            f, f1, g1 = out[nb]
            D.batch_fq(pos, sp, off, tabs[nb], 0.05, nb % 3, out=f)
            D.fq_grad(pos[:n1], sp[:n1], tabs[nb], 0.05, nb % 3, out_fq=f1,
                      out_grad=g1)

    def buffers():
        return {nb: (torch.empty((len(sizes), nb), device='cuda'),
                     torch.empty(nb, device='cuda'),
                     torch.empty((n1, 3, nb), device='cuda'))
                for nb in counts}

    want, got = buffers(), buffers()
    calls(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls(got)
    graph.replay()
    torch.cuda.synchronize()
    for nb in counts:
        assert all(torch.equal(a, b) for a, b in zip(want[nb], got[nb])), nb


def test_first_call_at_a_bin_count(D, ctx):
    """The first call at a bin count makes the window's tables for it: about
    0.1 ms of rotations at 1,300 bins and one copy beside 0.15 ms of what every
    such call does.  Three times that is the bound (sines and cosines instead
    of rotations take 1.5 ms)."""
    import time
    import torch
    pos, nums = particle(600, 5)
    sp = np.zeros(600, np.int32)
    pos = torch.as_tensor(pos, device='cuda')

    def call(nb):
        D.fq(pos, sp, np.ones((1, nb), np.float32), 0.02)
        torch.cuda.synchronize()

    call(1500)  # (workspaces)
    times = []
    for nb in range(1300, 1316):
        t = time.perf_counter()
        ran, _ = launched(ctx, 'fq', lambda: call(nb))
        times.append(time.perf_counter() - t)
        assert ran == 0
    assert np.median(times) <= 0.75e-3, times


@pytest.mark.parametrize('bad', [np.nan, np.inf])
def test_pair_force_of_a_lone_atom_without_a_place(D, ctx, bad):
    """A one-atom configuration has no pairs: its gradient is 0 wherever it
    is, and the other configurations' are untouched."""
    import torch
    e = O.update_experiment({'rstep': 0.02, 'rmax': 20.0})
    qb, rg = O.pdf_qbin(e), O.r_grid(e)
    nb = int(np.floor(e['qmax'] / qb))
    sizes = [300, 1, 65, 1, 280]
    pos = np.concatenate([particle(n, n)[0] for n in sizes])
    off = np.concatenate([[0], np.cumsum(sizes)])
    sp, tab, _ = species_tables([79] * len(pos), qb, nb)
    gobs = torch.as_tensor(O.pdf_fft(
        O.fq(S.fcc_nearest(4.0, 50).astype(np.float32),
             np.repeat(tab, 50, 0), qb), e['rstep'], qb, rg, e['qmin']))
    grads = []
    for x in (0.0, bad):
        pos[[300, 366], 1] = x
        ran, out = launched(ctx, 'adjoint', lambda: D.batch_potential_grad(
            pos, sp, off, tab, qb, e['rstep'], rg, e['qmin'], gobs))
        assert ran == 0
        grads.append(out['grad'].cpu().numpy())
    assert np.all(grads[1][[300, 366]] == 0)
    assert np.array_equal(grads[0], grads[1])
