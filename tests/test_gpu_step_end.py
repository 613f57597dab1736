"""The last launch of a device-loop step: it records the step in its own history slot and advances
the step counters, which every block of the launch reads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N(lesgpu_native, cuda_device):
    return lesgpu_native


def test_history_of_a_busy_gpu(N, tmp_path):
    """Probe lines of many warps a block, 120 steps, with another solver's launches between this
    one's: the files are the host-driven loop's, row for row, every tenth step's monitor row too."""
    from lesgpu.config import preset
    cfg = preset("tiny").replace(nx=24, ny=120, nz=8, lx=0.048, ly=0.24, lz=0.016, num_vortices=20,
                                 initial_flame_front_i=8, inlet_radius=0.008, seed=5)
    a, b = N.Solver(cfg), N.Solver(cfg)
    load = N.Solver(preset("c1"))
    da, db = tmp_path / "host", tmp_path / "device"
    for s, d in ((a, da), (b, db)):
        d.mkdir()
        s.set_outputs(str(d), N.LES_OUT_PROBES | N.LES_OUT_MONITOR)
    a.step(120)
    load.loop_begin(chunk=40)
    for _ in range(3):
        load.loop_run(40)
        b.run_device(40, chunk=40)
    for fn in ["simulation_monitor.csv"] + [f"probe_data_flame_region_loc{n}.csv" for n in range(7)]:
        assert (da / fn).exists() == (db / fn).exists()
        if (da / fn).exists():
            assert (da / fn).read_text() == (db / fn).read_text(), fn
    for f, x in a.state().items():
        np.testing.assert_array_equal(x, b.state()[f], err_msg=f)
    for s in (a, b, load):
        s.close()
