"""Tile gathers where their paths meet: tiles that stick out of the grid (odd
lengths), pairs of points whose stencils differ, boxes that are too large or
too wide to stage, rows that cannot be copied in 16-byte chunks, fields that
start off a 16-byte boundary, one and three fields, launches below and above
one wave of tiles, and values that are not finite."""
import numpy as np
import pytest

from oracle import claire_ref as R

pytestmark = pytest.mark.gpu

TOL = 1e-5  # transported images in single precision


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


def smooth(rng, shape, amp, kmax=3):
    x = R.grid_coords(shape)
    d = np.zeros((3,) + tuple(shape))
    for k in range(3):
        for _ in range(4):
            m = rng.integers(-kmax, kmax + 1, size=3)
            d[k] += rng.normal() * np.cos(sum(m[i] * x[i] for i in range(3)) + rng.uniform(0, 2 * np.pi))
    return (amp * d / np.abs(d).max()).astype(np.float32)


# (shape, largest displacement in cells): whole and partial tiles, floors that
# change inside a pair, boxes up to and beyond the staging limit
CASES = [((16, 16, 32), 0.4), ((17, 23, 36), 0.9), ((33, 9, 20), 1.7), ((40, 24, 52), 3.0), ((24, 40, 64), 9.0),
         ((21, 19, 30), 1.0), ((96, 80, 96), 2.5), ((97, 70, 100), 1.3),
         # strong maps: boxes that are staged only at the tight row pitch
         ((64, 64, 64), 6.0), ((72, 56, 96), 7.0)]


@pytest.mark.parametrize("shape,amp", CASES)
def test_interpolation(cb, shape, amp):
    rng = np.random.default_rng(sum(shape))
    disp = smooth(rng, shape, amp)
    q = R.index_grid(shape) + disp.astype(np.float64)
    f = rng.standard_normal((3,) + shape).astype(np.float32)
    ref = np.stack([R.interp3(f[k].astype(np.float64), q) for k in range(3)])
    out = cb.SemiLagrangian.Interpolate(to_dev(f), to_dev(disp)).cpu().numpy()
    assert rel(out, ref) < TOL
    one = cb.SemiLagrangian.Interpolate(to_dev(f[1]), to_dev(disp)).cpu().numpy()
    assert rel(one, ref[1]) < TOL


@pytest.mark.parametrize("shape,amp", CASES)
def test_one_field(cb, shape, amp):
    rng = np.random.default_rng(sum(shape) + 1)
    disp = smooth(rng, shape, amp)
    f = rng.standard_normal(shape).astype(np.float32)
    ref = R.interp3(f.astype(np.float64), R.index_grid(shape) + disp.astype(np.float64))
    out = cb.SemiLagrangian.Interpolate(to_dev(f), to_dev(disp)).cpu().numpy()
    assert rel(out, ref) < TOL


@pytest.mark.parametrize("shape,amp", [((16, 16, 32), 0.4), ((40, 24, 52), 3.0), ((97, 70, 100), 1.3)])
def test_field_off_a_16_byte_boundary(cb, shape, amp):
    import torch
    rng = np.random.default_rng(5)
    disp = smooth(rng, shape, amp)
    f = rng.standard_normal(shape).astype(np.float32)
    buf = torch.zeros(f.size + 1, device="cuda")
    buf[1:] = to_dev(f).ravel()
    out = cb.SemiLagrangian.Interpolate(buf[1:].view(shape), to_dev(disp)).cpu().numpy()
    assert rel(out, R.interp3(f.astype(np.float64), R.index_grid(shape) + disp.astype(np.float64))) < TOL


@pytest.mark.parametrize("shape", [(32, 32, 32), (96, 96, 96)])
def test_non_finite_values_stay_local(cb, shape):
    """A NaN reaches the points whose 64 taps hold it and no others."""
    rng = np.random.default_rng(11)
    disp = smooth(rng, shape, 0.8)
    f = rng.standard_normal(shape).astype(np.float32)
    f[5, 7, 9] = np.nan
    f[20, 20, 20] = np.inf
    out = cb.SemiLagrangian.Interpolate(to_dev(f), to_dev(disp)).cpu().numpy()
    base = [R.index_grid(shape)[k].astype(np.int64) + np.floor(disp[k]).astype(np.int64) - 1 for k in range(3)]
    hit = np.zeros(shape, bool)
    for p in ((5, 7, 9), (20, 20, 20)):
        inside = np.ones(shape, bool)
        for k in range(3):
            inside &= ((p[k] - base[k]) % shape[k]) < 4
        hit |= inside
    assert np.array_equal(~np.isfinite(out), hit)


@pytest.mark.parametrize("shape,amp", [((16, 48, 32), 0.5), ((96, 150, 64), 0.8), ((33, 26, 40), 0.3)])
def test_trajectory(cb, shape, amp):
    rng = np.random.default_rng(2)
    v = smooth(rng, shape, amp)
    for flag in ("state", "adjoint"):
        ref = R.trajectory_rk2(v.astype(np.float64), 4, flag)
        assert rel(cb.SemiLagrangian(4).ComputeTrajectory(to_dev(v), flag).cpu().numpy(), ref) < TOL
