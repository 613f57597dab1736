"""Attribute maps with fluid cells on the faces of the grid, which the reference never makes and the C ABI
takes: the stencils there read beside their field, so those cells' values mean nothing, but every
other cell's are what they are without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N(lesgpu_native, cuda_device):
    return lesgpu_native


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 4), (9, 12, 20), (12, 9, 17)])
def test_fluid_cells_on_every_face(N, nx, ny, nz, prec, staged):
    from lesgpu.config import preset
    cfg = preset("tiny").replace(nx=nx, ny=ny, nz=nz, lx=0.002 * nx, ly=0.002 * ny, lz=0.002 * nz, num_vortices=20,
                                 initial_flame_front_i=nx // 3, inlet_radius=0.001 * ny, seed=11)
    attr, st = N.initial_state(cfg)
    face = np.ones(attr.shape, dtype=bool)
    face[1:-1, 1:-1, 1:-1] = False
    out = []
    for a in (attr, np.where(face, 3, attr)):
        ctx = N.Context(cfg, precision=N.FP64 if prec == "fp64" else N.FP32)
        ctx.upload_attribute(a)
        ctx.upload_state(st)
        if staged and nz % (2 if prec == "fp64" else 4) == 0:
            ctx.set_scalar_staging(True)
        ctx.eval_rhs(600)
        out.append({k: ctx.field(k) for k in ["k_T", "k_G"] + [f"k_Y{s}" for s in range(5)]})
        ctx.close()
    # three cells of stencil and one of the filter
    deep = np.zeros(attr.shape, dtype=bool)
    deep[4:-4, 4:-4, 4:-4] = True
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k][deep], out[1][k][deep], err_msg=k)


def test_a_first_plane_of_fluid_reads_within_its_field(N):
    """Fields that are the same everywhere, all cells fluid: a cell of the first plane that reads beside its
    field would find another's values there.  No neighbour differs, so nothing but the nudging is left
    of the scalars' right-hand sides, the same on the first plane as inside."""
    from lesgpu.config import preset
    cfg = preset("tiny").replace(nx=8, ny=10, nz=12, lx=0.016, ly=0.02, lz=0.024, num_vortices=20,
                                 initial_flame_front_i=3, inlet_radius=0.005, seed=11)
    shape = (cfg.nx, cfg.ny, cfg.nz)
    ctx = N.Context(cfg)
    ctx.upload_attribute(np.full(shape, 3))
    level = {"u": -2.0, "v": -1.0, "w": -1.0, "T": 900.0, "G": 0.0, "rho": 0.4, "Y0": 0.05, "Y1": 0.2, "Y2": 0.7,
             "Y3": 0.03, "Y4": 0.02}
    ctx.upload_state({k: np.full(shape, v) for k, v in level.items()})
    ctx.eval_rhs(0)
    for k in ["k_T"] + [f"k_Y{s}" for s in range(5)]:
        x = ctx.field(k)[:-1, :-1, :-1]         # the last planes read what lies behind their field
        np.testing.assert_array_equal(x[0], np.broadcast_to(x[3, 3, 3], x[0].shape), err_msg=k)
    ctx.close()
