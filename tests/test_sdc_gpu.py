"""GPU parity of the density compensation estimate (estimate_dcw,
toolboxes/mri/sdc/SDC.hpp:19-80 with the Jinc kernel) against the oracle.
The device grids with float atomics and sums in float; the oracle sums in
FP64, hence relative-L2 tolerances."""
import numpy as np
import pytest
import torch

from gadgetron_b200 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

import gadgetron_b200 as gb  # noqa: E402


@pytest.mark.parametrize("N,os_factor,iters,kw", [((64, 64), 2.0, 10, 5.5), ((48, 80), 1.5, 5, 4.0),
                                                  ((64, 64), 3.0, 20, 5.5)])
def test_sdc_2d_matches_oracle(cuda, N, os_factor, iters, kw):
    traj = S.radial_golden_angle_2d(32, 128).astype(np.float32)
    w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), N, os_factor, iters, kw)
    ref = O.estimate_dcw(traj, N, os_factor, iters, kw)
    assert O.rel_l2(w.cpu().numpy(), ref) <= 1e-5


def test_sdc_3d_and_initial_weights(cuda):
    traj = S.kooshball_golden_means_3d(200, 32).astype(np.float32)
    init = S.ramp_dcw(traj).astype(np.float32)
    w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), (32, 32, 32), 2.0, 4, 4.0,
                            initial_dcw=torch.from_numpy(init).to(cuda))
    ref = O.estimate_dcw(traj, (32, 32, 32), 2.0, 4, 4.0, initial_dcw=init)
    assert O.rel_l2(w.cpu().numpy(), ref) <= 1e-5


def test_sdc_rejects_out_of_range(cuda):
    traj = torch.tensor([[0.2, 0.7]], dtype=torch.float32, device=cuda)
    with pytest.raises(gb.TrajectoryRangeError):
        gb.sdc.estimate_dcw(traj, (32, 32), 2.0, 2)


def test_sdc_repeated_calls_and_call_after_rejection(cuda):
    """Calls of changing grid sizes in turn, and a call after a rejected
    trajectory, reuse the kept scratch and still match the oracle."""
    small = S.radial_golden_angle_2d(16, 64).astype(np.float32)
    big = S.radial_golden_angle_2d(32, 128).astype(np.float32)
    cases = [(big, (96, 96)), (small, (32, 32)), (big, (96, 96))]
    for traj, N in cases:
        w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), N, 2.0, 5, 5.5)
        assert O.rel_l2(w.cpu().numpy(), O.estimate_dcw(traj, N, 2.0, 5, 5.5)) <= 1e-5
    bad = torch.tensor([[0.2, 0.7]], dtype=torch.float32, device=cuda)
    with pytest.raises(gb.TrajectoryRangeError):
        gb.sdc.estimate_dcw(bad, (32, 32), 2.0, 2)
    w = gb.sdc.estimate_dcw(torch.from_numpy(small).to(cuda), (32, 32), 2.0, 5, 5.5)
    assert O.rel_l2(w.cpu().numpy(), O.estimate_dcw(small, (32, 32), 2.0, 5, 5.5)) <= 1e-5


@pytest.mark.parametrize("M,kw,iters", [(1, 5.5, 2), (9, 0.95, 3), (777, 5.65, 2), (777, 5.8, 2), (777, 5.5, 1),
                                        (18945, 5.5, 2), (1 << 18, 2.0, 2), ((1 << 18) + 1, 2.0, 2)])
def test_sdc_2d_weight_table_limits(cuda, M, kw, iters):
    """Both sides of the weight table's limits: the smallest and widest square
    (2 x 2 and 11 x 11 taps), one wider, one iteration, a warp's second sample,
    and the largest sample count and one more."""
    traj = np.random.default_rng(M).uniform(-0.5, 0.5, (M, 2)).astype(np.float32)
    traj[0] = (-0.5, 0.5)
    w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), (48, 32), 2.0, iters, kw)
    assert O.rel_l2(w.cpu().numpy(), O.estimate_dcw(traj, (48, 32), 2.0, iters, kw)) <= 1e-5


def _square_sum32(u):
    """u0 * u0, then fused multiply-adds, each rounded to float32 (the double
    sums below are exact for offsets of whole float32 steps of the grid)."""
    d2 = u[..., 0] * u[..., 0]
    for d in range(1, u.shape[-1]):
        d2 = (u[..., d].astype(np.float64) ** 2 + d2).astype(np.float32)
    return d2


def _inside(d2, R, reciprocal):
    root = np.sqrt(d2)
    return (root * (np.float32(1.0) / R) if reciprocal else root / R) < np.float32(0.96960938)


def _edge_trajectory(D, mos, R, count):
    """Samples with a cell so close to the edge of their disc that sqrt(d2) / R
    and sqrt(d2) * (1 / R) put it on different sides, and as many whose cell is a
    step of the coordinate away from such a place."""
    rng = np.random.default_rng(D)
    half, limit = np.float32(mos // 2), float(np.float32(0.96960938) * R)
    out = []
    for _ in range(1000):
        if len(out) >= 2 * count:
            break
        n = 20000
        # coordinates in [16, 48) are multiples of 2^-18 of a cell, as k is of 2^-18 / mos
        step = 2.0 ** -18
        s = np.round(rng.uniform(17, 47, (n, D)) / step) * step
        cell = np.round(s)
        cell[:, 1] = np.floor(s[:, 1] - 1e-3)
        u = s - cell
        rest = limit ** 2 - np.sum(u ** 2, -1) + u[:, 1] ** 2
        keep = rest > 4.0
        s, cell = s[keep], cell[keep]
        # second coordinate so that the cell lies on the edge, a few steps either way
        cell[:, 1] = np.round(s[:, 1] - np.sqrt(rest[keep]))
        s[:, 1] = np.round((cell[:, 1] + np.sqrt(rest[keep])) / step) * step
        for k in range(-2, 3):
            t = s.copy()
            t[:, 1] += k * step
            u = (t - cell).astype(np.float32)
            d2 = _square_sum32(u)
            flips = _inside(d2, R, True) != _inside(d2, R, False)
            hit = t[flips & np.all((t > 16) & (t < 48), -1)]
            for row in hit[:max(0, count - len(out) // 2)]:
                out += [row, row + np.array([0.0, step] + [0.0] * (D - 2))]
    assert len(out) >= 2 * count
    k = ((np.array(out) - float(half)) / mos).astype(np.float32)
    assert np.array_equal(k.astype(np.float64) * mos + float(half), np.array(out))   # exact coordinates
    return k


def _estimate32(traj, mos, R, iters, reciprocal=False):
    """estimate_dcw with each tap's place decided in float32 as the kernel does
    (d2 by fused multiply-adds, root, division); weights and sums in double."""
    M, D = traj.shape
    s = (traj.astype(np.float64) * mos + mos // 2).astype(np.float32)
    lo = np.ceil(s - R).astype(np.int64)
    taps = np.stack(np.meshgrid(*[np.arange(int(2 * R) + 2)] * D, indexing="ij"), -1).reshape(-1, D)
    cells = lo[:, None] + taps[None]
    d2 = _square_sum32(s[:, None] - cells.astype(np.float32))
    r = (np.sqrt(d2) / R).astype(np.float64)
    w = np.maximum(sum(float(c) * r ** i for i, c in enumerate(O._JINC_C)), 0.0)
    w *= _inside(d2, R, reciprocal)
    idx = np.zeros(cells.shape[:2], np.int64)
    for d in range(D - 1, -1, -1):
        idx = idx * mos + np.mod(cells[..., d], mos)
    dcw = np.ones(M)
    for _ in range(iters):
        grid = np.bincount(idx.ravel(), weights=(w * dcw[:, None]).ravel(), minlength=mos ** D)
        dcw = dcw / np.sum(w * grid[idx], axis=1)
    return dcw


@pytest.mark.parametrize("D,iters", [(2, 1), (2, 4), (3, 2)])   # direct passes, weight table, direct 3D passes
def test_sdc_disc_edge_decided_by_the_quotient(cuda, D, iters):
    """The weight does not fall to zero where the disc ends, so a cell taken in
    or left out moves whole weights.  Tolerance: two float sums of positive
    terms and a quotient an iteration, rounding errors of 6e-8 each and of
    random sign; the other rule at the edge is off by more than ten times it."""
    # (width 4: there is a root that the two rules put on different sides; not every width has one)
    mos, R = 64, np.float32(np.float32(0.96960938) * np.float32(4.0))
    traj = _edge_trajectory(D, mos, R, 300)
    ref = _estimate32(traj, mos, R, iters)
    assert O.rel_l2(_estimate32(traj, mos, R, iters, reciprocal=True), ref) > 1e-5
    w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), (mos,) * D, 1.0, iters, 4.0)
    assert O.rel_l2(w.cpu().numpy(), ref) <= 1e-6


def test_sdc_keeps_one_large_grid(cuda):
    """A grid of more than 2^24 cells stays single: a call leaves no more device
    memory behind than that grid."""
    traj = S.kooshball_golden_means_3d(20, 32).astype(np.float32)
    n, cells = (256, 256, 512), 256 * 256 * 512
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    w = gb.sdc.estimate_dcw(torch.from_numpy(traj).to(cuda), n, 1.0, 2, 4.0)
    assert free - torch.cuda.mem_get_info()[0] < 1.5 * 4 * cells
    assert bool(torch.isfinite(w).all()) and bool((w > 0).all())
