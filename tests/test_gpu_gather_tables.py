"""Gathers with a box table (the solver's) at strong maps, and bf16 fields.

The time steps, the velocity at the feet, the cached gradients and the adjoint
factor read their tiles' boxes from a table.  At these velocities, 3 to 10 cells
a time step, tiles of all three kinds occur: boxes at the common row pitch, boxes
that only fit at the tight one, and boxes that are too large, which gather from
global memory.
"""
import numpy as np
import pytest

from oracle import claire_ref as R

pytestmark = pytest.mark.gpu

# A displacement of up to 10 cells carries about 1e-6 cells of roundoff; on images
# and velocities of wavenumber 3 and 4 that is under 1e-6 a step.  The gradient
# and the Hessian differentiate the warped images, whose spectrum reaches ten
# times further.
TOL_STATE, TOL_GRAD = 1e-5, 5e-5

CASES = [((64, 64, 64), 4.0), ((48, 64, 96), 6.0), ((64, 48, 32), 10.0)]


def rel(a, b):
    a = np.asarray(a, np.float64).ravel()
    b = np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module")
def cb(cuda):
    import claire_b200
    return claire_b200


def smooth(rng, shape, amp, kmax=3):
    x = R.grid_coords(shape)
    f = np.zeros(shape)
    for _ in range(4):
        m = rng.integers(-kmax, kmax + 1, size=3)
        f += rng.normal() * np.cos(sum(m[i] * x[i] for i in range(3)) + rng.uniform(0, 2 * np.pi))
    return amp * f / np.abs(f).max()


def problem(shape, amp, nt):
    """Images in [0, 1], a velocity of `amp` cells a time step, and a direction."""
    rng = np.random.default_rng(sum(shape))
    mR, mT = (0.5 + smooth(rng, shape, 0.5, 4) for _ in range(2))
    v = np.stack([smooth(rng, shape, amp * 2.0 * np.pi * nt / shape[k]) for k in range(3)])
    vt = np.stack([smooth(rng, shape, 1.0) for _ in range(3)])
    return [a.astype(np.float32) for a in (mR, mT, v, vt)]


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("shape,amp", CASES)
def test_solver_gathers(cb, shape, amp, bf16):
    nt = 2
    mR, mT, v, vt = problem(shape, amp, nt)
    prob = R.Problem(mR, mT, nt, R.Regularization("h1s", 1e-2), image_store=R.bf16_round if bf16 else None)
    g = prob.gradient(v.astype(np.float64))
    H = prob.hessian_matvec(vt.astype(np.float64))
    argv = ["-nx", "x".join(str(n) for n in shape), "-nt", str(nt), "-regnorm", "h1s", "-beta", "1e-2"]
    with cb.CLAIREInterface(cb.RegOpt(argv + (["-bf16images"] if bf16 else []))) as ci:
        ci.set_images(mR, mT)
        gg, Hg, m1 = ci.EvaluateGradient(v), ci.HessianMatVec(v, vt), ci.GetFinalState()
    # bf16: a value that roundoff moves across a rounding boundary changes by an ulp
    assert rel(m1, prob.solve_state()[nt]) < (1e-4 if bf16 else TOL_STATE)
    assert rel(gg, g) < (1e-3 if bf16 else TOL_GRAD)
    assert rel(Hg, H) < (1e-3 if bf16 else TOL_GRAD)


@pytest.mark.parametrize("shape,amp", CASES)
def test_bf16_field_is_the_fp32_gather_rounded(cb, shape, amp):
    import torch
    rng = np.random.default_rng(3)
    f = torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda().to(torch.bfloat16)
    disp = np.stack([smooth(rng, shape, amp) for _ in range(3)]).astype(np.float32)
    d = torch.from_numpy(disp).cuda()
    out = cb.SemiLagrangian.InterpolateBF16(f, d)
    assert torch.equal(out, cb.SemiLagrangian.Interpolate(f.float().contiguous(), d).to(torch.bfloat16))
    ref = R.interp3(f.float().cpu().numpy().astype(np.float64), R.index_grid(shape) + disp.astype(np.float64))
    assert rel(out.float().cpu().numpy(), ref) < 4e-3  # one bf16 rounding of the result
