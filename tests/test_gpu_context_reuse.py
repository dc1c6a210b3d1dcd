"""One context used for one call after another: what a call leaves behind (kept
scratch, captured graphs, CUDA's error state) must not reach the next one."""
import ctypes as C

import numpy as np
import pytest

from helpers import forestset
from lya2pcf_b200 import _native as N
from lya2pcf_b200.engine import PairEngine
from oracle import oracle as O
from test_gpu_edges import all_pairs, ragged

pytestmark = pytest.mark.gpu


def _check_distortion(eng, fs, f1, f2, np_, nt):
    D, W = eng.distortion()
    Do, Wo = O.distortion(fs, f1, f2, np_=np_, nt=nt)
    np.testing.assert_allclose(W, Wo, rtol=1e-12, atol=1e-12 * np.abs(Wo).max())
    assert np.abs(D - Do).max() <= 1e-10 * np.abs(Do).max() and np.abs(Do).max() > 0


def test_distortion_binnings_of_equal_size():
    """np x nt changed at equal np * nt: the rows of the column scratch get
    longer (and shorter again).  Tolerances of the other distortion tests."""
    fs = ragged(2.0)
    f1, f2 = all_pairs(fs)
    with PairEngine(np_=25, nt=64) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        for np_, nt in ((25, 64), (64, 25), (50, 32), (40, 40)):
            N.check(eng.lib.lya_set_bins(eng.ctx, 200.0, 200.0, np_, nt), eng.ctx)
            _check_distortion(eng, fs, f1, f2, np_, nt)


def test_distortion_long_forests_then_short():
    """Forests of 1500 pixels with the launch shape that takes them, then short
    ones on the same context with the default shape, which does not."""
    rng = np.random.default_rng(3)
    line = lambda L, k: dict(ra=0.5 + 0.01 * k, dec=0.1, dc=3600.0 + 0.9 * np.arange(L), w=rng.uniform(0.5, 2.0, L),  # noqa: E731
                             dw=rng.normal(0, 0.3, L))
    long = forestset([line(L, k) for k, L in enumerate((1500, 700))])
    short = forestset([line(L, k) for k, L in enumerate((90, 60, 33))])
    with PairEngine() as eng:
        for fs, shape in ((long, 4), (short, 0), (short, 4)):
            f1, f2 = all_pairs(fs)
            eng.upload(fs)
            eng.set_pairs(f1, f2)
            N.check(eng.lib.lya_dist_config(eng.ctx, shape, 0), eng.ctx)
            _check_distortion(eng, fs, f1, f2, 50, 50)


def test_a_refused_run_leaves_no_error_behind():
    """A binning beyond the shared memory is refused; the next calls, on this
    context and on a new one, are not."""
    fs = ragged(2.0)
    f1, f2 = all_pairs(fs)
    slot_start = np.searchsorted(fs.pix[f1], np.arange(fs.pix[-1] + 2))
    expect = O.corr(fs, f1, f2, slot_start)[1]

    def counts(eng):
        eng.run(kernel=N.KERNEL_FP64_DIAGONAL)
        return eng.histograms()[1]

    with PairEngine(np_=64, nt=64) as eng:
        eng.upload(fs)
        eng.set_pairs(f1, f2)
        for kernel in (N.KERNEL_FP32_GUARDED, N.KERNEL_FP64_DIAGONAL):
            with pytest.raises(N.LyaError):
                eng.run(kernel=kernel)
            with PairEngine() as other:
                other.upload(fs)
                other.set_pairs(f1, f2)
                assert np.array_equal(counts(other), expect)
            with pytest.raises(N.LyaError):
                eng.run(kernel=kernel)
            N.check(eng.lib.lya_set_bins(eng.ctx, 200.0, 200.0, 50, 50), eng.ctx)
            eng.nb = 2500
            assert np.array_equal(counts(eng), expect)
            N.check(eng.lib.lya_set_bins(eng.ctx, 200.0, 200.0, 64, 64), eng.ctx)


@pytest.mark.parametrize('nb_side', [50, 10])
def test_device_memory_as_a_host_output_is_refused(nb_side):
    """Device pointers where the library writes host results (of more and of
    less than 2 MB): an error status, and the context stays usable."""
    import torch
    nb = nb_side ** 2
    rng = np.random.default_rng(2)
    xi, w = rng.normal(size=(6, nb)), rng.uniform(1.0, 2.0, (6, nb))
    dev = torch.zeros(nb * nb, dtype=torch.float64, device='cuda')
    with PairEngine(np_=nb_side, nt=nb_side) as eng:
        mean, out, smooth = np.zeros(nb), np.zeros((nb, nb)), np.zeros((nb, nb))
        cov = lambda ptr: eng.lib.lya_covariance(eng.ctx, 6, N.ptr(xi), N.ptr(w), N.ptr(mean), ptr)  # noqa: E731
        N.check(cov(N.ptr(out)), eng.ctx)
        first = out.copy()
        assert cov(C.c_void_p(dev.data_ptr())) == 2
        out[:] = 0
        N.check(cov(N.ptr(out)), eng.ctx)
        np.testing.assert_array_equal(out, first)
        sm = C.c_int32(0)
        assert eng.lib.lya_covariance_smooth(eng.ctx, None, C.c_void_p(dev.data_ptr()), C.byref(sm)) == 2
        N.check(eng.lib.lya_covariance_smooth(eng.ctx, None, N.ptr(smooth), C.byref(sm)), eng.ctx)
        assert sm.value == 1 and np.isfinite(smooth).all()
    assert float(dev.abs().max()) == 0.0


def test_covariance_gives_large_row_scratch_back():
    """5,000 rows of 2,500 bins pass through 300 MB of device scratch, which an
    engine that lives on does not hold; 100 rows keep theirs (6 MB)."""
    import torch
    rng = np.random.default_rng(4)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    with PairEngine() as eng:
        mean, c = np.zeros(2500), np.zeros((2500, 2500))

        def cov(n):
            xi, w = rng.normal(size=(n, 2500)), rng.uniform(1.0, 2.0, (n, 2500))
            N.check(eng.lib.lya_covariance(eng.ctx, n, N.ptr(xi), N.ptr(w), N.ptr(mean), N.ptr(c)), eng.ctx)
            xm = (xi * w).sum(0) / w.sum(0)
            np.testing.assert_allclose(mean, xm, rtol=1e-12, atol=1e-14)
            y = w * (xi - xm)
            k = rng.integers(0, 2500, 40)
            np.testing.assert_allclose(c[np.ix_(k, k)], (y.T[k] @ y[:, k]) / np.outer(w.sum(0), w.sum(0))[np.ix_(k, k)],
                                       rtol=0, atol=1e-12 * np.abs(np.diag(c)).max())

        cov(100)
        before = free()
        cov(5000)
        assert free() >= before - (8 << 20)
        cov(100)
