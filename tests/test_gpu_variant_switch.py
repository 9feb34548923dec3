"""Sums over a transform's partials while another thread changes FFT variants.

A variant decides how many partials a reducing transform writes.  The variant
table is process-wide and other threads may change it between two calls into
the library's launchers (a server pool that tunes itself, claire_b200_autotune),
so the count that is summed has to be the one of the launch that wrote them.
Here a second thread changes the variants of all lengths all the time.
"""
import threading

import numpy as np
import pytest

from oracle import claire_ref as R

pytestmark = pytest.mark.gpu

# 72, 36 and 144 row CTAs a field at 48 points, and two column counts
N = 48


@pytest.fixture(scope="module")
def cb(cuda):
    import claire_b200
    return claire_b200


@pytest.fixture
def switching(cb):
    """Variants of N-point transforms change until the test ends."""
    stop = threading.Event()

    def flip():
        while not stop.is_set():
            for v in cb.fft_variant_candidates(N):
                cb.set_fft_variant(N, v)

    t = threading.Thread(target=flip)

    def start():
        t.start()

    yield start
    stop.set()
    if t.ident:
        t.join()
    cb.set_fft_variant(N, 0)


@pytest.mark.parametrize("norm", ["h1", "h2"])  # derivatives' partials, inverse transforms' partials
def test_functional(cb, switching, norm):
    import torch
    rng = np.random.default_rng(1)
    v = rng.standard_normal((3, N, N, N)).astype(np.float32)
    ref = R.Regularization(norm, 1e-2, 1e-4).functional(v.astype(np.float64))
    op, dv = cb.Regularization(norm, 1e-2, 1e-4), torch.from_numpy(v).cuda()
    switching()
    got = np.array([op.EvaluateFunctional(dv) for _ in range(300)])
    # single-precision transforms in any variant; a sum over too few partials
    # misses, over too many repeats, a fourth of them or more
    assert np.abs(got / ref - 1.0).max() < 1e-5


@pytest.mark.parametrize("graphs", ["0", "1"])
def test_registration(cb, switching, monkeypatch, graphs):
    """The PCG's dots are sums of the inverse transforms' partials."""
    monkeypatch.setenv("CLAIRE_B200_GRAPHS", graphs)
    mR, mT, _ = R.synthetic_c1(N, np.float64, 4)
    opt = cb.RegOpt(["-nx", str(N), "-nt", "4", "-regnorm", "h1s", "-beta", "1e-2", "-maxit", "2"])
    with cb.CLAIREInterface(opt) as ci:
        def solve():
            ci.set_images(mR.astype(np.float32), mT.astype(np.float32))
            ci.SetInitialGuess(np.zeros((3, N, N, N), np.float32))
            ci.Run()
            return ci.GetSolution().astype(np.float64), ci.stats()["pcg_iterations"]
        ref, its = solve()
        switching()
        for _ in range(4):
            v, k = solve()
            assert k == its
            # a seminorm: the solves differ by the rounding of the variants
            assert np.linalg.norm((v - ref).ravel()) < 1e-4 * np.linalg.norm(ref.ravel())
