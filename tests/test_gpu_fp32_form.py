"""The FP32 form's arithmetic is fixed operation by operation (csrc/les_f32_form.cuh): a run is the
run of the build its records were made with, and every kernel instance gives the same bits."""
import os
import sys

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu
sys.path.insert(0, GOLDEN)
import make_fp32_golden as M  # noqa: E402


@pytest.fixture(scope="module")
def N(lesgpu_native, cuda_device):
    return lesgpu_native


def _solver(N, case):
    nx, ny, nz, start = M.CASES[case]
    s = N.Solver(M.config(nx, ny, nz), precision=N.FP32, start_step=start)
    s.ctx.upload_state(M.state(nx, ny, nz, case == "ties"))
    return s


@pytest.mark.parametrize("case", list(M.CASES))
def test_run_is_the_recorded_run(N, case):
    """Twelve steps, every field to the last FP32 bit, before and after the WENO5 gradient sets in."""
    ref = np.load(os.path.join(GOLDEN, "fp32_ref.npz"))
    s = _solver(N, case)
    s.run(M.STEPS)
    for f, v in s.state().items():
        np.testing.assert_array_equal(v.astype(np.float32), ref[f"{case}_{f}"], err_msg=f)
    assert np.float32(s.last_dt) == np.float32(ref[f"{case}_dt"])
    s.close()


def test_flame_speeds_are_the_recorded_ones(N):
    """2e6 cells: the constant that keeps eta's divisor from zero changes five of their speeds."""
    assert M.speeds(N) == str(np.load(os.path.join(GOLDEN, "fp32_ref.npz"))["speeds"])


@pytest.mark.parametrize("case", list(M.CASES))
def test_every_instance_gives_the_same_bits(N, case):
    """Scalar and flow pass together and apart, 512-thread tiles, the staged scalar pass."""
    def tiles(t):
        return lambda s: s.ctx.set_tiles([0, t, t, t, 0])

    out = []
    for prepare in (lambda s: None, lambda s: s.ctx.kernel_timing(True), tiles(9), tiles(12),
                    lambda s: s.ctx.set_scalar_staging(M.CASES[case][2] % 4 == 0)):
        s = _solver(N, case)
        prepare(s)
        s.run(3)
        out.append(s.state())
        s.close()
    for q in out[1:]:
        for f, v in q.items():
            np.testing.assert_array_equal(v, out[0][f], err_msg=f)


@pytest.mark.parametrize("batched", [False, True])
def test_group_members_are_solo_runs(N, batched):
    """A member of a group and the run on its own, which on such a grid takes another kernel."""
    from lesgpu.ensemble import Ensemble
    nx, ny, nz, _ = M.CASES["early"]
    cfgs = [M.config(nx, ny, nz).replace(seed=11 + 7 * q) for q in range(3)]
    ens = Ensemble(cfgs, precision=N.FP32, autotune=False, batched=batched)
    for m in ens.members:
        m.ctx.upload_state(M.state(nx, ny, nz))
    ens.run(9, chunk=9)
    for c, m in zip(cfgs, ens.members):
        s = N.Solver(c, precision=N.FP32)
        s.ctx.upload_state(M.state(nx, ny, nz))
        s.run_device(9, chunk=9)
        assert s.last_dt == m.last_dt
        for f, v in m.state().items():
            np.testing.assert_array_equal(v, s.state()[f], err_msg=f)
        s.close()
    ens.close()
