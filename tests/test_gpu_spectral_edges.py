"""Transform kernels at the edges of their launch shapes: the shortest and the
longest axes, lengths whose butterflies do not fill a CTA (48, 96, 150, 192),
row and column counts that leave the last CTA partly empty, every FFT variant,
and derivative outputs that are not 8-byte aligned."""
import numpy as np
import pytest

from oracle import claire_ref as R

pytestmark = pytest.mark.gpu

# relative L2 error of single-precision transforms of these lengths
TOL = 1e-5


def rel(a, b):
    a = np.asarray(a, np.float64).ravel()
    b = np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module")
def cb(cuda):
    import claire_b200
    return claire_b200


def to_dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", [(16, 16, 16), (48, 150, 32), (150, 48, 96), (16, 32, 256), (256, 16, 48),
                                   (32, 192, 16), (192, 16, 192), (96, 64, 128)])
def test_every_axis_and_variant(cb, shape, variant):
    rng = np.random.default_rng(sum(shape))
    f = rng.standard_normal(shape).astype(np.float32)
    v = rng.standard_normal((3,) + shape).astype(np.float32)
    old = {n: cb.fft_variant(n) for n in shape}
    try:
        for n in shape:
            if variant in cb.fft_variant_candidates(n):
                cb.set_fft_variant(n, variant)
        assert rel(cb.fft_grad(to_dev(f)).cpu().numpy(), R.grad(f.astype(np.float64))) < TOL
        assert rel(cb.fft_div(to_dev(v)).cpu().numpy(), R.div(v.astype(np.float64))) < TOL
        for norm in ("h1s", "h1", "h2", "h3"):
            reg = R.Regularization(norm, 1e-2, 1e-1)
            op = cb.Regularization(norm, 1e-2, 1e-1)
            x = v.astype(np.float64)
            assert rel(op.EvaluateGradient(to_dev(v)).cpu().numpy(), reg.gradient(x)) < TOL, norm
            assert rel(op.ApplyInverse(to_dev(v)).cpu().numpy(), reg.apply_inverse(x)) < TOL, norm
            assert abs(op.EvaluateFunctional(to_dev(v)) / reg.functional(x) - 1.0) < TOL, norm
        for model in ("stokes", "relaxedstokes"):
            b = to_dev(v)
            cb.leray(b, model, (1e-2, 1e-4, 1e-4))
            assert rel(b.cpu().numpy(), R.leray_projection(v.astype(np.float64), model, 1e-2, 1e-4)) < TOL
    finally:
        for n, k in old.items():
            cb.set_fft_variant(n, k)


@pytest.mark.parametrize("shape", [(16, 32, 48), (64, 150, 16)])
def test_derivative_output_at_any_float(cb, shape):
    """An output that starts on an odd float takes 4-byte stores and the same values."""
    import torch
    rng = np.random.default_rng(3)
    f = to_dev(rng.standard_normal(shape))
    n = f.numel()
    ref = cb.fft_grad(f)
    buf = torch.zeros(3 * n + 1, device="cuda")
    cb.fft_grad(f, out=buf[1:].view((3,) + shape))
    assert torch.equal(buf[1:].view((3,) + shape), ref) and float(buf[0]) == 0.0
    v = to_dev(rng.standard_normal((3,) + shape))
    buf = torch.zeros(n + 1, device="cuda")
    cb.fft_div(v, out=buf[1:].view(shape))
    assert torch.equal(buf[1:].view(shape), cb.fft_div(v))
