"""The PCG's dots: summed in the inverse transforms' epilogues or in passes of
their own (CLAIRE_B200_FUSED_DOTS=0, read when a context is created).

Both sum the same single-precision products in FP64 in another order, so a
solve takes the same iterations and differs by single-precision roundoff of its
vectors (some 1e-7 each; 1e-5 here for two Gauss-Newton iterations).  The forms
differ by model and norm: without a projection the regularisation accumulates
into the body force, with one it adds it from another array, and the full norms
carry the regularised direction by recurrence instead of transforming it; one
batch mixes both.
"""
import numpy as np
import pytest

from oracle import claire_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cb(cuda):
    import claire_b200
    return claire_b200


@pytest.mark.parametrize("model", ["compressible", "stokes", "relaxedstokes"])
@pytest.mark.parametrize("norms", [("h1s",), ("h2",), ("h1s", "h2")])
def test_both_forms_take_the_same_solve(cb, monkeypatch, model, norms):
    n = 32
    mR, mT, _ = R.synthetic_c1(n, np.float64, 4)
    betas = {"h1s": "1e-2", "h2": "1e-3"}

    def opt(norm):
        o = cb.RegOpt(["-nx", str(n), "-nt", "4", "-regnorm", norm, "-beta", betas[norm], "-maxit", "2"])
        o.set("model", model)
        return o

    def solve(flag):
        monkeypatch.setenv("CLAIRE_B200_FUSED_DOTS", flag)
        with cb.CLAIREInterface(opt(norms[0]), nbatch=len(norms)) as ci:
            for b, norm in enumerate(norms):
                ci.set_problem_opts(b, opt(norm))
                ci.set_images(mR.astype(np.float32), mT.astype(np.float32), b)
            ci.Run()
            return [(ci.GetSolution(b).astype(np.float64), ci.stats(b)["pcg_iterations"]) for b in range(len(norms))]

    for (v1, k1), (v0, k0) in zip(solve("1"), solve("0")):
        assert k1 == k0 > 0
        assert np.linalg.norm((v1 - v0).ravel()) < 1e-5 * np.linalg.norm(v0.ravel()) > 0
