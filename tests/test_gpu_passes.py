"""The stage passes and the boundary kernel where they can go wrong: grids whose rows are no
multiple of a 16-byte access, grids as small as a solver takes, and cells on either side of the
line between the property pass's ordinary and general paths.

Tolerances: the parity tolerances of tests/test_gpu_parity.py (intermediates 1e-12, state 1e-10
after one step, 1e-8 after three).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "w", "T", "G", "rho", "Y0", "Y1", "Y2", "Y3", "Y4"]
PROPS = ["nu", "mu_mix", "Cp", "lambda", "alpha"] + [f"D{k}" for k in range(5)]


def rel(a, b):
    nb = np.linalg.norm(b)
    return float(np.linalg.norm(a - b) / (nb if nb > 0 else 1.0))


@pytest.fixture(scope="module")
def N(lesgpu_native, cuda_device):
    return lesgpu_native


def _grid(nx, ny, nz):
    from lesgpu.config import preset
    return preset("tiny").replace(nx=nx, ny=ny, nz=nz, lx=0.002 * nx, ly=0.002 * ny, lz=0.002 * nz,
                                  num_vortices=20, initial_flame_front_i=nx // 3, inlet_radius=0.5 * 0.002 * ny,
                                  seed=11)


@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 4), (5, 6, 7), (9, 8, 10), (12, 5, 33), (7, 9, 64), (16, 11, 130), (33, 7, 6)])
def test_steps_on_small_and_odd_grids(N, oracle_mod, nx, ny, nz):
    cfg = _grid(nx, ny, nz)
    orc = oracle_mod.Oracle(cfg.as_dict())
    sol = N.Solver(cfg)
    for n in (1, 2, 3):
        orc.step()
        sol.step()
        assert abs(sol.last_dt - orc.dt) <= 1e-13 * orc.dt, f"dt differs at step {n}"
        st, ref = sol.state(), orc.state()
        errs = {f: rel(st[f], ref[f]) for f in STATE}
        k = max(errs, key=errs.get)
        assert errs[k] <= (1e-10 if n == 1 else 1e-8), f"step {n}: {k} {errs[k]:.2e}"
    sol.close()
    orc.close()


@pytest.mark.parametrize("T", [140.0, 149.0, 151.0, 300.0, 999.0, 1001.0, 2200.0, 3990.0, 4100.0])
def test_properties_on_both_sides_of_the_ordinary_range(N, oracle_mod, T):
    """A temperature ramp of 3 per cent around T with every kind of composition: all species,
    several absent, one pure species, next to no mass."""
    cfg = _grid(17, 8, 12)
    orc = oracle_mod.Oracle(cfg.as_dict())
    shape = (cfg.nx, cfg.ny, cfg.nz)
    st = orc.state()
    i = np.arange(cfg.nx)[:, None, None] + np.zeros(shape)
    st["T"] = T * (0.985 + 0.03 * np.linspace(0.0, 1.0, cfg.nz)[None, None, :]) + np.zeros(shape)
    mixes = [[0.1, 0.2, 0.5, 0.12, 0.08], [0.0, 0.232, 0.768, 0.0, 0.0], [0.0, 0.0, 1.0, 0.0, 0.0],
             [0.06, 0.22, 0.72, 0.0, 0.0], [1e-14, 1e-14, 1e-14, 0.0, 0.0]]
    which = (i // 3).astype(int) % len(mixes)
    for k in range(5):
        st[f"Y{k}"] = np.array([m[k] for m in mixes])[which]
    st["rho"] = np.full(shape, 0.7)
    for f in STATE:
        orc.set_field(f, st[f])
    ctx = N.Context(cfg)
    ctx.upload_attribute(orc.attribute())
    ctx.upload_state(st)
    ctx.eval_rhs(0)
    orc.rhs_only(0)
    fluid = orc.attribute() == 3
    bad = {}
    for f in PROPS:
        e = rel(ctx.field(f)[fluid], orc.field(f)[fluid])
        if not e <= 1e-12:
            bad[f] = e
    ctx.close()
    orc.close()
    assert not bad, bad


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nz,tile", [(4, 4, 4, 0), (9, 8, 10, 7), (33, 7, 6, 6), (12, 5, 33, 3), (64, 32, 32, 0), (64, 32, 32, 2)])
def test_scalar_and_flow_in_one_launch(N, nx, ny, nz, tile, prec):
    """Small grids run the scalar and flow passes as halves of one block; with kernel timing on
    they run apart.  The arithmetic is the same: identical states in FP64, in FP32 up to how the
    compiler contracts it (2^-24 a term, 1e-6 over three steps)."""
    cfg = _grid(nx, ny, nz).replace(weno_transition_step=2)
    out = []
    for apart in (False, True):
        s = N.Solver(cfg, precision=N.FP64 if prec == "fp64" else N.FP32)
        s.ctx.set_tiles([0, tile, tile, tile, 0])
        s.ctx.kernel_timing(apart)
        s.step(3)
        out.append(s.state())
        s.close()
    for f in STATE:
        if prec == "fp64":
            np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
        else:
            assert rel(out[0][f], out[1][f]) <= 1e-6, f


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_dt_inputs_after_an_evaluation_are_that_states(N, prec):
    """An evaluation of the right-hand sides leaves the nu and alpha maxima of the state it evaluated,
    whatever larger ones the steps before it left."""
    cfg = _grid(16, 11, 20)
    s = N.Solver(cfg, precision=N.FP64 if prec == "fp64" else N.FP32)
    s.step(2)
    umax, nu0, al0 = s.ctx.dt_inputs()
    st = s.state()
    st["T"] = 0.5 * (st["T"] + st["T"].min())       # colder, so less viscous
    st["rho"] = st["rho"] * 1.5
    s.ctx.upload_state(st)
    assert N.lib().lesgpu_set_dt_inputs(s.ctx._h, nu0, al0) == 0
    s.ctx.eval_rhs(0)
    _, nu, al = s.ctx.dt_inputs()
    fluid = s.attribute() == 3
    assert nu == s.field("nu")[fluid].max() < nu0
    assert al == s.field("alpha")[fluid].max() < al0
    s.close()


@pytest.mark.parametrize("rho", [0.0, 0.7])
def test_density_of_cells_without_mass_fractions(N, oracle_mod, rho):
    """Where the mass fractions are all zero the step keeps the density through its stages and the
    sweep after the boundary conditions sets 1.2, whatever the density was, zero included."""
    cfg = _grid(17, 12, 14).replace(relax=0.0)
    orc = oracle_mod.Oracle(cfg.as_dict())
    sol = N.Solver(cfg)
    shape = (cfg.nx, cfg.ny, cfg.nz)
    st = orc.state()
    for f in STATE:
        st[f] = np.full(shape, {"T": 300.0, "rho": rho}.get(f, 0.0))
        orc.set_field(f, st[f])
    sol.ctx.upload_state(st)
    orc.step()
    sol.step()
    got, want = sol.state()["rho"], orc.state()["rho"]
    assert (want[5:-3, 3:-3, 3:-3] == 1.2).all()
    np.testing.assert_allclose(got, want, rtol=1e-10)
    sol.close()
    orc.close()


@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 4), (5, 6, 7), (33, 7, 6), (12, 9, 40)])
def test_faces_copy_mass_fractions_before_they_are_renormalised(N, nx, ny, nz):
    """Open faces copy a cell's mass fractions as the last stage leaves them, and the sweep after the
    boundary conditions divides the cell's own by their sum: an outflow cell of the k-faces, divided by
    its sum, is its neighbour to the last bit."""
    cfg = _grid(nx, ny, nz)
    s = N.Solver(cfg)
    st = s.state()
    rng = np.random.default_rng(2)
    for f, a in (("u", 3.0), ("v", 1.0), ("w", 4.0)):
        st[f] = a * rng.standard_normal(st[f].shape)
    y = rng.uniform(0.02, 1.0, (5,) + st["u"].shape)
    for k in range(5):
        st[f"Y{k}"] = y[k] / y.sum(0)
    s.ctx.upload_state(st)
    s.step(1)
    st = s.state()
    attr = s.attribute()
    n = 0
    for face, near, out in ((0, 1, st["w"][:, :, 1] <= 0), (nz - 1, nz - 2, st["w"][:, :, nz - 2] >= 0)):
        m = out & (attr[:, :, face] == 4) & (attr[:, :, near] == 3)
        m[[0, -1]] = m[:, [0, -1]] = False
        Y = [st[f"Y{k}"][:, :, face][m] for k in range(5)]
        total = (((Y[0] + Y[1]) + Y[2]) + Y[3]) + Y[4]
        for k in range(5):
            np.testing.assert_array_equal(Y[k] / total, st[f"Y{k}"][:, :, near][m])
        n += int(m.sum())
    assert n > 0
    s.close()


def test_wide_tiles_leave_a_small_grid_its_launch_shape(N):
    """A small grid runs the scalar and flow pass in one launch of 256-thread tiles.  Where the tiles set
    for the two passes have 512, it takes the grid's default, not the first of the table, whose padding
    costs a fifth of the step on 60x20x40: no more than a tenth above the time without any tiles set."""
    import time
    from lesgpu.config import preset
    cfg = preset("c1").replace(nx=60, ny=20, nz=40, num_vortices=50, initial_flame_front_i=15)
    best = []
    for tiles in (None, 9):
        s = N.Solver(cfg)
        if tiles:
            d = s.ctx.get_tiles()
            s.ctx.set_tiles([d[0], d[1], tiles, tiles, d[4]])
        s.loop_begin(chunk=200)
        s.loop_run(200)
        t = []
        for _ in range(7):
            t0 = time.perf_counter()
            s.loop_run(200)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
        s.close()
    assert best[1] <= 1.1 * best[0], best


@pytest.mark.parametrize("seed", [1, 2])
def test_property_routines_against_cudas_own(N, seed):
    """The reciprocal (2^-60 and its rounding) and the corrected quotient (half a unit and a rounding) are at most
    a last place from the correctly rounded ones; the exponential is within 1.1 last places and CUDA's
    exp2 within one; FP32 quotients by normal denominators have the approximate division's bits."""
    rcp, ex, quot, differ = N.selfcheck_math(1 << 26, seed)
    assert rcp <= 1.0 and quot <= 1.0
    assert ex <= 2.1
    assert differ == 0
