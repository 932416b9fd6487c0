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
