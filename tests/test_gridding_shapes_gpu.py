"""The gridding kernel over the forms its dispatch chooses between: coil counts
around every coil group (1 to 33), 2D and 3D, plain and compensated sums,
tiles with no samples and tiles split into chunks, samples that are not
finite, and the fixed-scratch entry point's two chunk lengths.
Against the oracle (float weights, double sums): relative L2 <= PARITY_TOL."""
import ctypes

import numpy as np
import pytest
import torch

from gadgetron_b200 import synthetic as S
from oracle import oracle as O
from tests.helpers import PARITY_TOL, footprint_cells, rel_l2

pytestmark = pytest.mark.gpu

import gadgetron_b200 as gb  # noqa: E402
from gadgetron_b200._lib import lib  # noqa: E402

COILS = [1, 2, 3, 4, 5, 8, 9, 12, 16, 17, 24, 33]


def _samples(coils, m, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((coils, m)) + 1j * rng.standard_normal((coils, m))).astype(np.complex64)


def _adjoint_and_normal(N, mos, W, traj, coils, flags, cuda):
    D = len(N)
    plan = gb.NFFT.make_plan(N, mos, W, flags=flags)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, D))
    y = _samples(coils, traj.shape[0], coils)
    w = S.ramp_dcw(traj)
    wt = torch.from_numpy(w).to(cuda)
    x = torch.empty((coils, 1) + tuple(reversed(N)), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, wt, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    ref = orc.backwards_nc2c(y, w[None])
    assert rel_l2(x.cpu().numpy(), ref) <= PARITY_TOL
    img = S.gaussian_image((coils, 1) + tuple(reversed(N)), coils + 1)
    nrm = torch.empty_like(x)
    plan.mult_MH_M(torch.from_numpy(img).to(cuda), nrm, wt)
    assert rel_l2(nrm.cpu().numpy(), orc.mult_MH_M(img, w[None])) <= PARITY_TOL
    assert plan.device_errors() == 0


@pytest.mark.parametrize("coils", COILS)
@pytest.mark.parametrize("W,alpha", [(5.5, 2.0), (4.0, 1.5)])
def test_2d_coil_groups(cuda, coils, W, alpha):
    """64 spokes through one centre (split tiles) on a rectangular grid."""
    N = (64, 32)
    mos = tuple(-(-int(n * alpha) // 32) * 32 for n in N)
    _adjoint_and_normal(N, mos, W, S.radial_golden_angle_2d(64, 96), coils, 0, cuda)


@pytest.mark.parametrize("coils", [1, 3, 8, 12, 17])
def test_2d_compensated(cuda, coils):
    _adjoint_and_normal((64, 64), (96, 96), 4.0, S.radial_golden_angle_2d(70, 96), coils, gb.FLAG_COMPENSATED, cuda)


@pytest.mark.parametrize("coils", [1, 2, 4, 7, 16, 20])
@pytest.mark.parametrize("flags", [0, 1])
def test_3d_coil_groups(cuda, coils, flags):
    N, mos = (32, 64, 32), (64, 96, 64)
    _adjoint_and_normal(N, mos, 4.0, S.kooshball_golden_means_3d(300, 48), coils, flags, cuda)


def test_wide_form_of_16_coils(cuda):
    """Enough frames that the 16-coil gridding takes its wide form; the same
    frames in a plan of their own take the narrow one."""
    N, mos, W, C, F = (64, 64), (128, 128), 5.5, 16, 40
    trajs = [S.radial_golden_angle_2d(8 + f % 5, 64, profile_offset=13 * f) for f in range(F)]
    offs = np.cumsum([0] + [t.shape[0] for t in trajs]).tolist()
    y = _samples(C, offs[-1], 3)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(np.concatenate(trajs)).to(cuda), frame_offsets=offs)
    x = torch.empty((C, F, 64, 64), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    for f in (0, 17, 39):
        orc = O.OraclePlan(N, mos, W)
        orc.preprocess(trajs[f][None])
        ref = orc.backwards_nc2c(y[:, offs[f]:offs[f + 1]])
        assert rel_l2(x[:, f].cpu().numpy(), ref[:, 0]) <= PARITY_TOL, f


def _series(coils, frames, seed):
    """Short radial frames of 64^2 on 128^2 and their samples."""
    trajs = [S.radial_golden_angle_2d(5 + f % 3, 64, profile_offset=13 * f) for f in range(frames)]
    offs = np.cumsum([0] + [t.shape[0] for t in trajs]).tolist()
    return trajs, offs, _samples(coils, offs[-1], seed)


@pytest.mark.parametrize("tile", [(32, 16), (16, 32), (64, 8), (32, 32), (16, 8), (8, 16)])
@pytest.mark.parametrize("coils", [16, 32])
def test_wide_form_on_every_tile(cuda, tile, coils):
    """Enough frames for the wide 16-coil form (14208 bricks of the narrow one)
    on tiles of 128 to 1024 cells: 2 to 16 bricks a tile, one or several CTAs."""
    N, mos, W = (64, 64), (128, 128), 5.5
    bricks = tile[0] // 4 * (tile[1] // 8)
    F = -(-14208 * 16 // (coils * bricks * (128 * 128 // (tile[0] * tile[1]))))
    trajs, offs, y = _series(coils, F, 3)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.set_tiling(tile, 16)
    plan.preprocess(torch.from_numpy(np.concatenate(trajs)).to(cuda), frame_offsets=offs)
    x = torch.empty((coils, F, 64, 64), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    for f in (0, F // 2, F - 1):
        orc = O.OraclePlan(N, mos, W)
        orc.preprocess(trajs[f][None])
        ref = orc.backwards_nc2c(y[:, offs[f]:offs[f + 1]])
        assert rel_l2(x[:, f].cpu().numpy(), ref[:, 0]) <= PARITY_TOL, f


@pytest.mark.parametrize("group", [4, 8, 16])
@pytest.mark.parametrize("tile", [(16, 16), (32, 16), (16, 32), (32, 32), (8, 32), (32, 8), (8, 8, 4), (8, 8, 8),
                                  (16, 8, 8), (8, 16, 8), (16, 16, 4)])
def test_every_tile_of_the_autotuner(cuda, tile, group):
    """Every tile and coil group that the autotuner times, both directions of
    17 coils against the oracle."""
    D, coils = len(tile), 17
    N, mos = ((32, 64), (64, 96)) if D == 2 else ((32, 32, 32), (64, 64, 64))
    traj = S.radial_golden_angle_2d(40, 96) if D == 2 else S.kooshball_golden_means_3d(80, 48)
    plan = gb.NFFT.make_plan(N, mos, 4.0)
    plan.set_tiling(tile, group)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, 4.0)
    orc.preprocess(traj.reshape(1, -1, D))
    y = _samples(coils, traj.shape[0], group)
    x = torch.empty((coils, 1) + tuple(reversed(N)), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    assert rel_l2(x.cpu().numpy(), orc.backwards_nc2c(y)) <= PARITY_TOL
    img = S.gaussian_image((coils, 1) + tuple(reversed(N)), 3)
    out = torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(img).to(cuda), out, None, gb.NFFT_comp_mode.FORWARDS_C2NC)
    assert rel_l2(out.cpu().numpy(), orc.forward_c2nc(img)) <= PARITY_TOL


@pytest.mark.parametrize("coils", [9, 12, 24])
def test_wide_forms_of_other_coil_counts(cuda, coils):
    """The wide form with idle coils, and the 12-coil form, which takes over at
    the same launch size; a frame by itself takes the narrow form."""
    N, mos, W = (64, 64), (128, 128), 5.5
    F = -(-14208 // (64 * 8 * -(-coils // 16)))
    trajs, offs, y = _series(coils, F, 4)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(np.concatenate(trajs)).to(cuda), frame_offsets=offs)
    x = torch.empty((coils, F, 64, 64), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    for f in (0, F - 1):
        one = gb.NFFT.make_plan(N, mos, W)
        one.preprocess(torch.from_numpy(trajs[f]).to(cuda))
        xo = torch.empty((coils, 1, 64, 64), dtype=torch.complex64, device=cuda)
        yf = np.ascontiguousarray(y[:, offs[f]:offs[f + 1]])
        one.compute(torch.from_numpy(yf).to(cuda), xo, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
        orc = O.OraclePlan(N, mos, W)
        orc.preprocess(trajs[f][None])
        ref = orc.backwards_nc2c(yf)[:, 0]
        assert rel_l2(x[:, f].cpu().numpy(), ref) <= PARITY_TOL
        assert rel_l2(xo[:, 0].cpu().numpy(), ref) <= PARITY_TOL


@pytest.mark.parametrize("coils", [8, 12, 16, 18])
@pytest.mark.parametrize("W", [4.0, 5.5])
def test_long_lists(cuda, coils, W):
    """Thousands of samples to a tile: lists cut into chunks of 512, two bricks
    per CTA with several warps to a brick."""
    _adjoint_and_normal((32, 32), (64, 64), W, S.radial_golden_angle_2d(150, 200), coils, 0, cuda)


@pytest.mark.parametrize("coils,m", [(9, 32767), (9, 32768), (16, 33000), (20, 33000)])
def test_convolve_on_two_streams(cuda, coils, m):
    """The standalone gridding from the caller's array and, from 32768 samples
    and 9 coils on, through the plan's rows: calls on two streams in turn, then
    one under capture, give the same as the oracle."""
    N, mos, W = (64, 64), (128, 128), 4.0
    traj = np.random.default_rng(m).uniform(-0.5, 0.5, (m, 2)).astype(np.float32)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj[None])
    ys = [_samples(coils, m, s) for s in (1, 2)]
    yt = [torch.from_numpy(y).to(cuda) for y in ys]
    out = [torch.empty((coils, 1) + mos, dtype=torch.complex64, device=cuda) for _ in ys]
    plan.convolve(yt[0], out[0], gb.NFFT_conv_mode.NC2C)   # allocations before the overlap
    streams = [torch.cuda.Stream() for _ in ys]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, y, o in zip(streams, yt, out):
            with torch.cuda.stream(s):
                plan.convolve(y, o, gb.NFFT_conv_mode.NC2C)
    torch.cuda.synchronize()
    refs = [orc.convolve_nc2c(y) for y in ys]
    for o, r in zip(out, refs):
        assert rel_l2(o.cpu().numpy(), r) <= PARITY_TOL
    graph = torch.cuda.CUDAGraph()
    out[0].zero_()
    with torch.cuda.graph(graph):
        plan.convolve(yt[0], out[0], gb.NFFT_conv_mode.NC2C)
    graph.replay()
    torch.cuda.synchronize()
    assert rel_l2(out[0].cpu().numpy(), refs[0]) <= PARITY_TOL


def test_3d_four_slices_of_8_coils(cuda):
    """More than 4 M (tile, sample) pairs: the four-slice form of 5 to 8 coils."""
    N, mos, W, coils = (32, 32, 32), (64, 64, 64), 4.0, 5
    traj = np.random.default_rng(2).uniform(-0.5, 0.5, (1400000, 3)).astype(np.float32)
    y = _samples(coils, traj.shape[0], 6)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    g = torch.empty((coils, 1) + mos, dtype=torch.complex64, device=cuda)
    plan.convolve(torch.from_numpy(y).to(cuda), g, gb.NFFT_conv_mode.NC2C)
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, 3))
    assert rel_l2(g.cpu().numpy(), orc.convolve_nc2c(y)) <= PARITY_TOL


def test_autotune_of_a_16_coil_series(cuda):
    """The autotuner times every candidate tile on a launch of the wide form,
    and leaves a plan that reconstructs."""
    N, mos, W, C, F = (64, 64), (128, 128), 5.5, 16, 30
    trajs, offs, y = _series(C, F, 5)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(np.concatenate(trajs)).to(cuda), frame_offsets=offs)
    plan.autotune(C)
    x = torch.empty((C, F, 64, 64), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(trajs[7][None])
    assert rel_l2(x[:, 7].cpu().numpy(), orc.backwards_nc2c(y[:, offs[7]:offs[8]])[:, 0]) <= PARITY_TOL


@pytest.mark.parametrize("group", [1, 2, 4])
@pytest.mark.parametrize("coils", [4, 5, 17])
@pytest.mark.parametrize("D", [2, 3])
def test_coil_groups_smaller_than_the_coil_count(cuda, D, coils, group):
    """A coil group set by the caller, on both sides of the coil count from
    which the adjoint lays its samples into rows; every direction."""
    N, mos, tile = ((64, 32), (128, 64), (16, 16)) if D == 2 else ((32, 32, 32), (64, 64, 64), (8, 8, 8))
    traj = S.radial_golden_angle_2d(24, 96) if D == 2 else S.kooshball_golden_means_3d(60, 48)
    plan = gb.NFFT.make_plan(N, mos, 4.0)
    plan.set_tiling(tile, group)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, 4.0)
    orc.preprocess(traj.reshape(1, -1, D))
    y, w = _samples(coils, traj.shape[0], coils), S.ramp_dcw(traj)
    img = S.gaussian_image((coils, 1) + tuple(reversed(N)), 7)
    it, wt = torch.from_numpy(img).to(cuda), torch.from_numpy(w).to(cuda)
    x, out = torch.empty_like(it), torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, wt, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    assert rel_l2(x.cpu().numpy(), orc.backwards_nc2c(y, w[None])) <= PARITY_TOL
    plan.compute(it, out, None, gb.NFFT_comp_mode.FORWARDS_C2NC)
    assert rel_l2(out.cpu().numpy(), orc.forward_c2nc(img)) <= PARITY_TOL
    plan.mult_MH_M(it, x, wt)
    assert rel_l2(x.cpu().numpy(), orc.mult_MH_M(img, w[None])) <= PARITY_TOL


@pytest.mark.parametrize("coils", [1, 2, 4, 8, 12, 16])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite_sample_stays_in_its_footprint(cuda, coils, bad):
    N, mos, W = (64, 64), (128, 128), 5.5
    traj = S.radial_golden_angle_2d(24, 128)
    y = _samples(coils, traj.shape[0], 9)
    j = 1700
    y[coils - 1, j] = bad
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    grid = torch.empty((coils, 1, 128, 128), dtype=torch.complex64, device=cuda)
    plan.convolve(torch.from_numpy(y).to(cuda), grid, gb.NFFT_conv_mode.NC2C)
    g = grid.cpu().numpy()[:, 0]
    hit = footprint_cells(traj[j], mos, W)
    assert np.all(np.isfinite(g[:coils - 1]))
    assert np.all(np.isfinite(g[coils - 1][~hit]))
    assert not np.any(np.isfinite(g[coils - 1][hit]))


def test_noalloc_long_chunks_when_the_short_ones_do_not_fit(cuda):
    """Dense centre, many coils: the partial tiles of the short chunks exceed
    the fixed 16 MiB scratch, those of the long chunks do not; the call is
    accepted and equals the regular entry point."""
    N, mos, W, C = (128, 128), (256, 256), 5.5, 64
    traj = S.radial_golden_angle_2d(256, 256)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    y = torch.from_numpy(_samples(C, traj.shape[0], 2)).to(cuda)
    ref = torch.empty((C, 1, 256, 256), dtype=torch.complex64, device=cuda)
    plan.convolve(y, ref, gb.NFFT_conv_mode.NC2C)
    out = torch.full_like(ref, float("nan"))
    accepted = 0
    for nb in (1, 8, 16, 32, 64):
        st = lib.gb_nufft_convolve_nc2c_noalloc(plan._h, ctypes.c_void_p(y.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                                0, nb, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st == 0:
            accepted = nb
            assert rel_l2(out[:nb].cpu().numpy(), ref[:nb].cpu().numpy()) <= PARITY_TOL
    assert accepted >= 8


def test_noalloc_groups_larger_than_the_scratch(cuda):
    """48 coils in 3D run as two groups of 32 and need the scratch of 64; where
    48 coils' partial tiles fit and 64 coils' do not, the call is accepted and
    runs on fewer coils at a time."""
    N, mos, W, C = (32, 32, 32), (64, 64, 64), 4.0, 64
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def noalloc(plan, y, out, nb):
        return lib.gb_nufft_convolve_nc2c_noalloc(plan._h, ctypes.c_void_p(y.data_ptr()),
                                                  ctypes.c_void_p(out.data_ptr()), 0, nb, stream)

    for spokes in range(40, 600, 20):
        traj = S.kooshball_golden_means_3d(spokes, 48)
        plan = gb.NFFT.make_plan(N, mos, W)
        plan.preprocess(torch.from_numpy(traj).to(cuda))
        y = torch.from_numpy(_samples(C, traj.shape[0], 2)).to(cuda)
        out = torch.full((C, 1) + mos, float("nan"), dtype=torch.complex64, device=cuda)
        if noalloc(plan, y, out, 48) == 0 and noalloc(plan, y, out, 64) == 1:
            ref = torch.empty((48, 1) + mos, dtype=torch.complex64, device=cuda)
            plan.convolve(y[:48].contiguous(), ref, gb.NFFT_conv_mode.NC2C)
            assert rel_l2(out[:48].cpu().numpy(), ref.cpu().numpy()) <= PARITY_TOL
            return
    pytest.fail("no trajectory between the two scratch sizes")
