"""Preprocess at sample counts around its run and tile lengths (warp runs of
128, 256 and 512 elements, tiles of 1024 to 4096, scans of 16384 counts), with
empty frames and frames of one sample: both directions against the oracle
(relative L2 <= PARITY_TOL), and a second preprocess of the same plan and the
same results bit for bit from a new one."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import PARITY_TOL, rel_l2

pytestmark = pytest.mark.gpu

import gadgetron_b200 as gb  # noqa: E402


@pytest.mark.parametrize("m", [1, 31, 33, 1023, 1025, 8192, 32767, 32769, 131071, 131073])
def test_sample_counts(cuda, m):
    rng = np.random.default_rng(m)
    N, mos, W = (64, 32), (96, 64), 4.0
    traj = rng.uniform(-0.5, 0.5, (m, 2)).astype(np.float32)
    traj[: m // 2] *= 0.2   # half of them crowd around the centre
    y = (rng.standard_normal((2, m)) + 1j * rng.standard_normal((2, m))).astype(np.complex64)
    t = torch.from_numpy(traj).to(cuda)
    x, outs = torch.empty((2, 1, 32, 64), dtype=torch.complex64, device=cuda), []
    for fresh in range(2):
        plan = gb.NFFT.make_plan(N, mos, W)
        for _ in range(1 + 3 * fresh):   # eager, recorded and replayed segments
            plan.preprocess(t)
        plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
        back = torch.empty((2, m), dtype=torch.complex64, device=cuda)
        plan.compute(x, back, None, gb.NFFT_comp_mode.FORWARDS_C2NC)
        outs.append((x.cpu().numpy(), back.cpu().numpy()))
    orc = O.OraclePlan(N, mos, W)
    orc.preprocess(traj[None])
    ref = orc.backwards_nc2c(y)
    assert rel_l2(outs[0][0], ref) <= PARITY_TOL
    assert rel_l2(outs[0][1], orc.forward_c2nc(outs[0][0])) <= PARITY_TOL
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])


def test_empty_and_single_sample_frames(cuda):
    rng = np.random.default_rng(5)
    N, mos, W = (32, 32), (64, 64), 5.5
    sizes = [0, 1, 700, 0, 33, 1]
    offs = np.cumsum([0] + sizes).tolist()
    traj = rng.uniform(-0.5, 0.5, (offs[-1], 2)).astype(np.float32)
    y = (rng.standard_normal((3, offs[-1])) + 1j * rng.standard_normal((3, offs[-1]))).astype(np.complex64)
    plan = gb.NFFT.make_plan(N, mos, W)
    plan.preprocess(torch.from_numpy(traj).to(cuda), frame_offsets=offs)
    x = torch.empty((3, len(sizes), 32, 32), dtype=torch.complex64, device=cuda)
    plan.compute(torch.from_numpy(y).to(cuda), x, None, gb.NFFT_comp_mode.BACKWARDS_NC2C)
    x = x.cpu().numpy()
    for f, m in enumerate(sizes):
        if m == 0:
            assert not x[:, f].any()
            continue
        orc = O.OraclePlan(N, mos, W)
        orc.preprocess(traj[offs[f]:offs[f + 1]][None])
        ref = orc.backwards_nc2c(np.ascontiguousarray(y[:, offs[f]:offs[f + 1]]))
        assert rel_l2(x[:, f], ref[:, 0]) <= PARITY_TOL, f
