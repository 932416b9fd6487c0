"""The project-written FFT passes at the lengths with a factor 7, 9 or 15 (16 x
14, 18, 28, 30, 36): NUFFT in both directions with pruned and unpruned spans,
2D and 3D, and the row-fused CG iteration, against the oracle (relative L2 <=
PARITY_TOL, CG <= 1e-4)."""
import numpy as np
import pytest
import torch

from gadgetron_b200 import synthetic as S
from oracle import oracle as O
from tests.helpers import PARITY_TOL, rel_l2

pytestmark = pytest.mark.gpu

import gadgetron_b200 as gb  # noqa: E402


def _check(cuda, N, mos, W, traj, coils, flags=0):
    D = len(N)
    dcw = S.ramp_dcw(traj)
    dt = torch.from_numpy(dcw).to(cuda)
    plan = gb.NFFT.make_plan(N, mos, W, flags=flags)
    plan.preprocess(torch.from_numpy(traj).to(cuda))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj.reshape(1, -1, D))
    img = S.gaussian_image((coils, 1) + tuple(reversed(N)), 3)
    x = torch.from_numpy(img).to(cuda)
    y = torch.empty((coils, traj.shape[0]), dtype=torch.complex64, device=cuda)
    plan.compute(x, y, dt, gb.NFFT_comp_mode.FORWARDS_C2NC)
    ref = orc.forward_c2nc(img, dcw.reshape(1, -1))
    assert rel_l2(y.cpu().numpy(), ref) <= PARITY_TOL
    back = torch.empty_like(x)
    plan.compute(y, back, dt, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    assert rel_l2(back.cpu().numpy(), orc.backwards_nc2c(ref, dcw.reshape(1, -1))) <= PARITY_TOL
    full = torch.empty((coils, 1) + tuple(reversed(mos)), dtype=torch.complex64, device=cuda)
    plan.compute(y, full, dt, gb.NFFT_comp_mode.BACKWARDS_NC2C)   # oversampled image: no pruning
    assert rel_l2(full.cpu().numpy(), orc.backwards_nc2c(ref, dcw.reshape(1, -1), oversampled_out=True)) <= PARITY_TOL


@pytest.mark.parametrize("N,mos", [((128, 160), (224, 288)), ((224, 128), (448, 256)), ((320, 224), (480, 288)),
                                   ((288, 384), (576, 480)), ((192, 352), (288, 448)), ((32, 288), (64, 576))])
def test_2d(cuda, N, mos):
    _check(cuda, N, mos, 4.0, S.radial_golden_angle_2d(24, 96), 2)


def test_3d(cuda):
    _check(cuda, (32, 64, 32), (64, 288, 224), 4.0, S.kooshball_golden_means_3d(150, 48), 2)


@pytest.mark.parametrize("N,mos,W,frames", [((192, 128), (288, 224), 4.0, 1), ((96, 224), (192, 448), 5.5, 2)])
def test_cg(cuda, N, mos, W, frames):
    coils = 5
    trajs = [S.radial_golden_angle_2d(24 + 7 * f, 128, profile_offset=11 * f) for f in range(frames)]
    offs = np.cumsum([0] + [t.shape[0] for t in trajs]).tolist()
    sq = np.concatenate([np.sqrt(S.ramp_dcw(t)) for t in trajs]).astype(np.float32)
    csm = S.gaussian_bump_csm(tuple(reversed(N)), coils)
    ph = S.ellipse_phantom(tuple(reversed(N)), 12, 4)
    E = gb.cuNonCartesianSenseOperator(2)
    E.setup(N, mos, W)
    E.set_csm(torch.from_numpy(csm).to(cuda))
    E.set_dcw(torch.from_numpy(sq).to(cuda))
    E.preprocess(torch.from_numpy(np.concatenate(trajs)).to(cuda), frame_offsets=offs)
    d, refs = np.zeros((coils, offs[-1]), np.complex64), []
    for f in range(frames):
        P = O.OraclePlan(N, mos, W)
        P.preprocess(trajs[f][None])
        op = O.OracleSense(P, csm, sq[offs[f]:offs[f + 1]][None])
        d[:, offs[f]:offs[f + 1]] = op.mult_M(ph[None]).reshape(coils, -1)
        refs.append(O.cg_solve(op, d[:, offs[f]:offs[f + 1]][:, None, :], iterations=5, tc_tolerance=0.0)[0])
    cg = gb.cuCgSolver()
    cg.set_encoding_operator(E)
    cg.set_max_iterations(5)
    cg.set_tc_tolerance(0.0)
    cg.set_frame_independent(True)
    for fused in (True, False):
        cg.set_row_fusion(fused)
        x = cg.solve(torch.from_numpy(d).to(cuda)).cpu().numpy()
        for f in range(frames):
            assert rel_l2(x[f], refs[f]) <= 1e-4, (fused, f)
    assert E.get_plan().device_errors() == 0
