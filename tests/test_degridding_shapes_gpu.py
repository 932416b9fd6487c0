"""The table degridding and the trajectory gradient over the forms their
dispatch chooses between: coil counts around every coil group (1 to 33), 2D and
3D, plain and compensated sums, and cells that are not finite.  Degridding
against the oracle (float weights, double sums): relative L2 <= PARITY_TOL."""
import numpy as np
import pytest
import torch

from gadgetron_b200 import synthetic as S
from oracle import oracle as O
from tests.helpers import PARITY_TOL, footprint_cells, rel_l2

pytestmark = pytest.mark.gpu

import gadgetron_b200 as gb  # noqa: E402


def _samples(coils, m, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((coils, m)) + 1j * rng.standard_normal((coils, m))).astype(np.complex64)


@pytest.mark.parametrize("coils", [1, 2, 3, 4, 5, 8, 9, 12, 16, 17, 24, 33])
@pytest.mark.parametrize("D,W,alpha,flags", [(2, 5.5, 2.0, 0), (2, 4.0, 1.5, 0), (2, 4.0, 1.5, 1), (2, 6.0, 2.0, 0),
                                             (3, 4.0, 1.5, 0), (3, 4.0, 1.5, 1)])
def test_forward_coil_groups(cuda, D, W, alpha, flags, coils):
    N = (64, 32, 64)[:D]
    mos = tuple(-(-int(n * alpha) // 32) * 32 for n in N)
    traj = S.radial_golden_angle_2d(40, 97) if D == 2 else S.kooshball_golden_means_3d(120, 47)
    plan = gb.NFFT.make_plan(N, mos, W, flags=gb.FLAG_COMPENSATED if flags else 0)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, D))
    img = S.gaussian_image((coils, 1) + tuple(reversed(N)), coils + 1)
    out = torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(img).to(cuda), out, None, gb.NFFT_comp_mode.FORWARDS_C2NC)
    assert rel_l2(out.cpu().numpy(), orc.forward_c2nc(img)) <= PARITY_TOL


@pytest.mark.parametrize("coils", [1, 2, 4, 8, 12, 16])
def test_nonfinite_cell_reaches_only_samples_over_it(cuda, coils):
    N, mos, W = (64, 64), (128, 128), 5.5
    traj = S.radial_golden_angle_2d(24, 128)
    rng = np.random.default_rng(4)
    g = (rng.standard_normal((coils, 1, 128, 128)) + 1j * rng.standard_normal((coils, 1, 128, 128))).astype(np.complex64)
    y0, x0 = 70, 57
    g[0, 0, y0, x0] = np.nan
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    out = torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.convolve(torch.from_numpy(g).to(cuda), out, gb.NFFT_conv_mode.C2NC)
    y = out.cpu().numpy()
    over = np.array([footprint_cells(k, mos, W)[y0, x0] for k in traj])
    assert np.array_equal(~np.isfinite(y[0]), over)
    assert np.all(np.isfinite(y[1:]))


@pytest.mark.parametrize("coils", [3, 17, 33])
@pytest.mark.parametrize("D", [2, 3])
def test_trajectory_gradient_adds_over_coils(cuda, D, coils):
    """The gradient of all coils (coil groups of 4, 8 or 16 in turn) is the sum
    of the single coils' (each in a group of one)."""
    if D == 2:
        N, mos, W, traj = (64, 32), (96, 64), 4.0, S.radial_golden_angle_2d(40, 96)
    else:
        N, mos, W, traj = (32, 32, 32), (64, 64, 64), 4.0, S.kooshball_golden_means_3d(150, 48)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    img = torch.from_numpy(S.gaussian_image((coils, 1) + tuple(reversed(N)), 5)).to(cuda)
    w = torch.from_numpy(_samples(coils, traj.shape[0], 6)).to(cuda)
    dcw = torch.from_numpy(S.ramp_dcw(traj)).to(cuda)
    total = plan.traj_grad(img, w, dcw)
    one = sum(plan.traj_grad(img[c:c + 1].contiguous(), w[c:c + 1].contiguous(), dcw).double() for c in range(coils))
    # 32-bit sums of W^D taps and `coils` coils in another order
    assert rel_l2(total.cpu().numpy(), one.cpu().numpy()) <= 2e-6


def _first_tap_trajectory(D, W, mos):
    """Samples whose first cell comes out differently from the padded and from
    the unpadded float coordinate along some dimension, random along the others."""
    r, hw = np.float32(W) * np.float32(0.5), int(np.ceil(W / 2))
    bias = float((mos + 2 * hw) >> 1)
    odd = []
    for p in (16.0, 32.0, 64.0, 128.0):   # every float of the padded coordinate just above a power of two
        c = np.arange(p, p + hw, 2.0 ** -23 * p).astype(np.float32)
        c = c[np.ceil(c - r) != np.ceil((c - np.float32(hw)) - r) + hw]
        k = ((c.astype(np.float64) - bias) / mos).astype(np.float32)
        odd += k[((k.astype(np.float64) * mos + bias).astype(np.float32) == c) & (np.abs(k) < 0.5)].tolist()
    assert odd
    rng = np.random.default_rng(int(10 * W))
    traj = rng.uniform(-0.5, 0.5, (64 * D, D)).astype(np.float32)
    for d in range(D):
        traj[64 * d:64 * (d + 1), d] = rng.choice(odd, 64)
    return traj


@pytest.mark.parametrize("D,W,flags", [(1, 5.3, 0), (2, 5.3, 0), (2, 5.3, 1), (2, 3.7, 0), (2, 2.7, 0), (3, 5.3, 0),
                                       (3, 4.6, 1)])
@pytest.mark.parametrize("coils", [1, 2, 16])
def test_first_tap_where_float_grids_differ(cuda, D, W, flags, coils):
    """Just above a power of two the padded coordinate's floats are coarser than
    the unpadded one's; the taps have to start where the weight table does."""
    N, mos = ((64,) * D, (128,) * D) if D < 3 else ((32,) * D, (64,) * D)
    traj = _first_tap_trajectory(D, W, mos[0])
    plan = gb.NFFT.make_plan(N, mos, W, flags=gb.FLAG_COMPENSATED if flags else 0)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, D))
    rng = np.random.default_rng(1)
    g = (rng.standard_normal((coils, 1) + mos) + 1j * rng.standard_normal((coils, 1) + mos)).astype(np.complex64)
    w = _samples(coils, traj.shape[0], 2)
    out = torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.convolve(torch.from_numpy(g).to(cuda), out, gb.NFFT_conv_mode.C2NC)
    assert rel_l2(out.cpu().numpy(), orc.convolve_c2nc(g)) <= PARITY_TOL
    grad = plan.traj_grad_from_grid(torch.from_numpy(g).to(cuda), torch.from_numpy(w).to(cuda))
    assert rel_l2(grad.cpu().numpy(), orc.traj_grad_from_grid(g, w)) <= PARITY_TOL


def _kinds(a):
    """-1, 1: that infinity; 2: NaN; 0: finite."""
    return np.where(np.isnan(a), 2, np.where(np.isinf(a), np.sign(a), 0)).astype(int)


@pytest.mark.parametrize("coils", [1, 2, 4, 8, 12, 16])
@pytest.mark.parametrize("D,W", [(2, 5.5), (2, 4.0), (3, 4.0)])
def test_infinite_cell_gives_infinite_samples(cuda, D, W, coils):
    """Footprints have floor(W) or floor(W) + 1 taps a dimension; in the shorter
    ones no cell may be read with a weight of zero (0 * inf)."""
    N, mos = (32,) * D, (64,) * D
    rng = np.random.default_rng(8)
    traj = rng.uniform(-0.08, 0.08, (600, D)).astype(np.float32)
    g = (rng.standard_normal((coils, 1) + mos) + 1j * rng.standard_normal((coils, 1) + mos)).astype(np.complex64)
    g.real[(0, 0) + (30,) * D] = -np.inf
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    out = torch.empty((coils, 600), dtype=torch.complex64, device=cuda)
    plan.convolve(torch.from_numpy(g).to(cuda), out, gb.NFFT_conv_mode.C2NC)
    y = out.cpu().numpy()
    over = np.array([footprint_cells(k, mos, W)[(30,) * D] for k in traj])
    assert over.sum() >= 20
    assert np.array_equal(_kinds(y.real[0]), -1 * over)
    assert np.all(np.isfinite(y.imag)) and np.all(np.isfinite(y[1:]))
    # the gradient: infinite with the sign of the weights' derivative
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, D))
    w = np.ones((coils, 600), np.complex64)
    grad = plan.traj_grad_from_grid(torch.from_numpy(g).to(cuda), torch.from_numpy(w).to(cuda)).cpu().numpy()
    big = np.where(np.isinf(g.real), np.float32(-1e30), g.real) + 1j * g.imag
    sign = np.sign(orc.traj_grad_from_grid(big, w))
    assert np.array_equal(_kinds(grad), np.where(over[:, None], sign, 0))
