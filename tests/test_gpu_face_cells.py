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
