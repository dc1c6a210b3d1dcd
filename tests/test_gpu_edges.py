"""Kernels that walk the exact bin edges of sorted forests, against the oracle's
per-pair reference formula, where a walk can go wrong: forest lengths around
the 32- and 64-pixel chunks, pixels exactly on rp edges, pixel steps below and
above a bin, bins so narrow in rt that a row meets many edges, one bin only,
binnings that leave the walk to the general kernel, and forests that do."""
import numpy as np
import pytest

from helpers import forestset
from lya2pcf_b200 import _native as N
from lya2pcf_b200.engine import PairEngine
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = (1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 200, 330, 614)


def ragged(step, unsorted=False, seed=5):
    """Forests of LENGTHS pixels within half a degree, some coincident lines of
    sight; distances on a common grid (so that differences fall exactly on rp
    edges for coincident lines of sight) and a jittered copy of it."""
    rng = np.random.default_rng(seed)
    grid = 3600.0 + step * np.arange(1200) - 1e-4 * step * np.arange(1200) ** 2 / 8
    exact = 3600.0 + step * np.arange(1200)
    forests = []
    for k, L in enumerate(LENGTHS):
        o = int(rng.integers(0, 500))
        dc = (exact if k % 3 == 0 else grid)[o:o + L].copy()
        if k % 3 == 1:
            dc += rng.uniform(0, 0.4 * step)
        if unsorted and k % 4 == 2 and L > 2:
            dc = dc[::-1].copy()
        ra, dec = (0.5, 0.1) if k % 5 == 0 else (0.5 + rng.uniform(0, 0.03), 0.1 + rng.uniform(-0.02, 0.02))
        forests.append(dict(ra=ra + 1e-9 * k, dec=dec, dc=dc, w=rng.uniform(0.5, 2.0, L), dw=rng.normal(0, 0.3, L),
                            z=2.0 + 1e-3 * np.arange(L)))
    return forestset(forests, pix=np.arange(len(LENGTHS)) // 6)


def all_pairs(fs):
    f1, f2 = np.triu_indices(fs.n, 1)
    return f1.astype(np.int32), f2.astype(np.int32)


BINNINGS = [
    (50, 50, 2.0, False),      # steps of half an rp bin
    (50, 50, 2.0, True),       # some forests unsorted: the general kernel for their pairs
    (50, 50, 9.0, False),      # steps above a bin
    (200, 16, 2.0, False),     # the same from narrow rp bins
    (16, 200, 2.0, False),     # a row meets many rt edges
    (1, 1, 2.0, False),
    (64, 64, 2.0, False),      # largest binning of 64 rp bins
    (4096, 1, 0.5, False),     # too many rp edges for shared memory
]


@pytest.mark.parametrize('np_,nt,step,unsorted', BINNINGS)
def test_adjoint_edges(np_, nt, step, unsorted):
    """Gradient against the oracle.  Both add the same products (<= 15 x 614
    per pixel) in FP64 in different orders: 1e4 x 2^-53 of the largest
    component's terms, 1e-11 of the largest component allowed."""
    fs = ragged(step, unsorted)
    f1, f2 = all_pairs(fs)
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        eng.run(kernel=N.KERNEL_FP64_PLAIN)
        W, DW = eng.totals()
        g = np.random.default_rng(7).normal(size=eng.nb)
        gdw, gw = eng.adjoint(g)
    cdw = np.divide(g, W, out=np.zeros_like(W), where=W != 0)
    odw, ow = O.adjoint(fs, f1, f2, cdw, -cdw * np.divide(DW, W, out=np.zeros_like(W), where=W != 0), np_=np_, nt=nt)
    assert np.abs(odw).max() > 0
    np.testing.assert_allclose(gdw, odw, rtol=0, atol=1e-11 * np.abs(odw).max())
    np.testing.assert_allclose(gw, ow, rtol=0, atol=1e-11 * np.abs(ow).max())


@pytest.mark.parametrize('np_,nt,step,unsorted', [(50, 50, 2.0, False), (50, 50, 2.0, True), (50, 50, 9.0, False),
                                                  (64, 16, 2.0, False), (33, 20, 2.0, False), (31, 20, 2.0, False),
                                                  (1, 1, 2.0, False)])
def test_distortion_edges(np_, nt, step, unsorted):
    """D and W against the oracle's eta products: the tolerance of the other
    distortion tests (1e-10 of max|D|, W to 1e-12)."""
    fs = ragged(step, unsorted)
    f1, f2 = all_pairs(fs)
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        D, W = eng.distortion()
    Do, Wo = O.distortion(fs, f1, f2, np_=np_, nt=nt)
    np.testing.assert_allclose(W, Wo, rtol=1e-12, atol=1e-12 * np.abs(Wo).max())
    assert np.abs(D - Do).max() <= 1e-10 * np.abs(Do).max() and np.abs(Do).max() > 0


@pytest.mark.parametrize('np_,nt,step,unsorted', [
    (50, 50, 2.0, False), (50, 50, 2.0, True), (50, 50, 9.0, False), (200, 12, 2.0, False), (12, 200, 2.0, False),
    (1, 1, 2.0, False), (300, 8, 2.0, False),
    (600, 4, 2.0, False)])   # the last: edge tables beyond the shared memory, the one-diagonal walk
def test_fp64_walk_edges(np_, nt, step, unsorted):
    """FP64 kernel against the oracle: counts equal, sums to 1e-12 (DW to 1e-12
    of the sum of the moduli), as in the other FP64 tests."""
    fs = ragged(step, unsorted)
    f1, f2 = all_pairs(fs)
    slot_start = np.searchsorted(fs.pix[f1], np.arange(fs.pix[-1] + 2))
    hist, cnt = O.corr(fs, f1, f2, slot_start, np_=np_, nt=nt)
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        for run_cap in (0, 8):
            eng.run(kernel=N.KERNEL_FP64_DIAGONAL, run_cap=run_cap)
            h, c = eng.histograms()
            assert np.array_equal(c, cnt) and cnt.sum() > 0
            for q in (N.Q_W, N.Q_DW, N.Q_RP, N.Q_RT, N.Q_Z):
                scale = hist[:, O.Q_DWABS if q == N.Q_DW else q]
                assert np.all(np.abs(h[:, q] - hist[:, q]) <= 1e-12 * scale), q


@pytest.mark.parametrize('unsorted', [False, True])
@pytest.mark.parametrize('np_,nt,fits', [(53, 52, True), (47, 59, True), (53, 53, False), (64, 44, False)])
def test_fp64_binnings_taken(np_, nt, fits, unsorted):
    """Binnings around the shared memory's limit are taken or refused whatever
    the forests are; a refused one leaves the context usable."""
    fs = ragged(2.0, unsorted)
    f1, f2 = all_pairs(fs)
    slot_start = np.searchsorted(fs.pix[f1], np.arange(fs.pix[-1] + 2))
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        if not fits:
            with pytest.raises(N.LyaError):
                eng.run(kernel=N.KERNEL_FP64_DIAGONAL)
            np_ = nt = 50
            N.check(eng.lib.lya_set_bins(eng.ctx, 200.0, 200.0, np_, nt), eng.ctx)
            eng.nb = np_ * nt
        eng.run(kernel=N.KERNEL_FP64_DIAGONAL)
        _, c = eng.histograms()
    assert np.array_equal(c, O.corr(fs, f1, f2, slot_start, np_=np_, nt=nt)[1])


@pytest.mark.parametrize('np_,nt,where', [(50, 72, 'lean'), (37, 100, 'lean'), (37, 23, 'negative'), (50, 50, 'negative'),
                                          (64, 60, 'far'), (31, 50, 'far')])
def test_distortion_sorted_forests_of_the_general_builder(np_, nt, where):
    """Sorted forests whose columns are not built from edges: more than 64 rt
    bins, or distances that are negative or above 1e6.  Same tolerances."""
    fs = ragged(2.0)
    if where == 'negative':
        for f in range(fs.n):
            a, b = int(fs.start[f]), int(fs.start[f + 1])
            fs.dc[a:b] -= fs.dc[a] + 50.0
    elif where == 'far':
        fs.dc += 1e6
    f1, f2 = all_pairs(fs)
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        D, W = eng.distortion()
    Do, Wo = O.distortion(fs, f1, f2, np_=np_, nt=nt)
    np.testing.assert_allclose(W, Wo, rtol=1e-12, atol=1e-12 * np.abs(Wo).max())
    assert np.abs(D - Do).max() <= 1e-10 * np.abs(Do).max() and np.abs(Do).max() > 0


def lines(lengths, masked, seed=8):
    """A forest of every length, within a quarter degree, steps of 2 Mpc/h; with
    `masked`, each lacks a stretch of pixels in its middle."""
    rng = np.random.default_rng(seed)
    forests = []
    for L in lengths:
        dc = 3700.0 + 2.0 * np.arange(L) + rng.uniform(0, 60.0)
        if masked:
            dc[L // 2:] += 31.0
        forests.append(dict(ra=0.5 + rng.uniform(0, 4e-3), dec=0.1 + rng.uniform(0, 4e-3), dc=dc,
                            w=rng.uniform(0.5, 2.0, L), dw=rng.normal(0, 0.3, L), z=2.0 + 1e-3 * np.arange(L)))
    # and one that is not sorted: the walks of sorted forests leave its pairs to a second kernel
    forests.append(dict(forests[0], dc=np.array([3702.0, 3700.0]), w=np.ones(2), dw=np.ones(2), z=np.full(2, 2.0)))
    return forestset(forests, pix=np.arange(len(forests)) // 8)


@pytest.mark.parametrize('lengths,np_,nt,masked,exact', [
    ((13,) * 12, 50, 50, False, True), ((13,) * 11 + (12,), 50, 50, False, False),
    ((22, 23) * 6, 12, 200, False, False), ((23,) * 12, 12, 200, False, True),
    ((120,) * 12, 200, 12, False, True), ((120,) * 12, 200, 12, True, False), ((120,) * 12, 100, 20, True, True),
    ((120, 3) * 6, 400, 4, True, False), ((614, 1) * 3, 50, 50, True, True)])
def test_fp64_walk_chosen(lengths, np_, nt, masked, exact):
    """Short forests, and masked ones in narrow rp bins, take the one-diagonal
    walk, which serves the unsorted forest in the same launch; counts and sums of
    either as in test_fp64_walk_edges."""
    fs = lines(lengths, masked)
    f1, f2 = all_pairs(fs)
    slot_start = np.searchsorted(fs.pix[f1], np.arange(fs.pix[-1] + 2))
    hist, cnt = O.corr(fs, f1, f2, slot_start, np_=np_, nt=nt)
    launches = {}
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        for variant in (1, 0):
            for _ in range(2):
                before = eng.stats()['launches']
                launches[variant] = eng.run(kernel=N.KERNEL_FP64_DIAGONAL, variant=variant)['launches'] - before
            h, c = eng.histograms()
            np.testing.assert_array_equal(c, cnt)
            for q in (N.Q_W, N.Q_RP, N.Q_RT, N.Q_Z):
                np.testing.assert_allclose(h[:, q], hist[:, q], rtol=1e-12, atol=0)
    assert launches[0] - launches[1] == (1 if exact else 0)


@pytest.mark.parametrize('lengths,np_,nt,masked,band', [
    ((36,) * 12, 50, 50, False, True), ((36,) * 11 + (35,), 50, 50, False, False),
    ((112,) * 12, 200, 12, False, False), ((114,) * 12, 200, 12, False, True), ((300,) * 6, 250, 10, False, False),
    ((130,) * 8, 10, 300, False, True), ((130,) * 8, 10, 300, True, False), ((614, 1) * 3, 4, 600, False, False),
    ((120,) * 12, 50, 50, True, False), ((120,) * 12, 40, 40, True, True), ((120,) * 12, 64, 64, True, True),
    ((120,) * 12, 200, 20, True, False), ((20,) * 12, 64, 64, False, True), ((20,) * 11 + (19,), 64, 64, False, False)])
def test_adjoint_kernel_chosen(lengths, np_, nt, masked, band):
    """Short forests, narrow rp bins and masked forests take the gather kernel,
    which serves the unsorted forest in the same launch; gradients of either as
    in test_adjoint_edges."""
    fs = lines(lengths, masked)
    f1, f2 = all_pairs(fs)
    with PairEngine(np_=np_, nt=nt) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        eng.run(kernel=N.KERNEL_FP64_PLAIN)
        W, DW = eng.totals()
        g = np.random.default_rng(7).normal(size=eng.nb)
        for _ in range(2):
            before = eng.stats()['launches']
            gdw, gw = eng.adjoint(g)
            launches = eng.stats()['launches'] - before
    cdw = np.divide(g, W, out=np.zeros_like(W), where=W != 0)
    odw, ow = O.adjoint(fs, f1, f2, cdw, -cdw * np.divide(DW, W, out=np.zeros_like(W), where=W != 0), np_=np_, nt=nt)
    assert np.abs(odw).max() > 0
    np.testing.assert_allclose(gdw, odw, rtol=0, atol=1e-11 * np.abs(odw).max())
    np.testing.assert_allclose(gw, ow, rtol=0, atol=1e-11 * np.abs(ow).max())
    assert launches == (5 if band else 4)   # coefficients, pair kernels, two copies
