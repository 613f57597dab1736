"""States of the FP32 form, written by the build of the library that LESGPU_LIB names (a B200):

    LESGPU_LIB=<build>/liblesgpu.so python tests/golden/make_fp32_golden.py

fp32_ref.npz holds what tests/test_gpu_fp32_form.py compares with: the fields after STEPS steps of
each case, rounded to FP32, and the SHA-256 of a field of flame speeds.  It was written by the first FP32 build whose runs were compared with
the FP64 form's (the operations of csrc/les_f32_form.cuh, left to the compiler to contract).
"""
import hashlib
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(HERE)), "combustion-les-optimization_b200"))

CASES = {"early": (22, 13, 17, 0), "late": (24, 12, 16, 600), "ties": (20, 14, 18, 0)}
STEPS = 12


def config(nx, ny, nz):
    from lesgpu.config import preset
    return preset("tiny").replace(nx=nx, ny=ny, nz=nz, lx=0.002 * nx, ly=0.002 * ny, lz=0.002 * nz, num_vortices=20,
                                  initial_flame_front_i=nx // 3, inlet_radius=0.001 * ny, seed=11)


def state(nx, ny, nz, spikes=False):
    """A front through a swirling flow, formed with additions, products and quotients only, so that it
    is the same to the last bit everywhere; with `spikes`, single cells off a level G, whose stencils tie."""
    x, y, z = (np.arange(n).reshape([-1 if q == d else 1 for q in range(3)]) / n for d, n in enumerate((nx, ny, nz)))
    z = z - 0.5
    r = 9.0 * (y - 0.35 + 0.3 * x * x + 0.4 * z * z - 0.5 * x * z) + 0.0 * (x + y + z)
    g = np.clip(0.5 + 0.65 * r / (1.0 + np.abs(r)), 0.0, 1.0)
    if spikes:
        i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
        g = 0.5 + np.where((i % 5 == 2) & (j % 5 == 2) & (k % 5 == 2), ((7 * i + 3 * j + 5 * k) % 13 - 6) / 256.0, 0.0)
    st = {"u": 14.0 * (1.0 - 1.6 * y) + 20.0 * z * (x - 0.4), "v": 9.0 * (z * 2.0 - y + 0.3) * (1.2 - x),
          "w": 11.0 * (0.4 - y - z * x), "G": g, "T": 300.0 + 1900.0 * g}
    ys = [0.06 * (1.0 - g), 0.22 - 0.215 * g, 0.72 + 0.0 * g, 0.175 * g, 0.095 * g]
    total = ys[0] + ys[1] + ys[2] + ys[3] + ys[4]
    ys = [q / total for q in ys]
    w = [0.0440956, 0.0319988, 0.0280134, 0.0440095, 0.0180153]
    st["rho"] = 101325.0 / (8.314462 * (ys[0] / w[0] + ys[1] / w[1] + ys[2] / w[2] + ys[3] / w[3] + ys[4] / w[4]) * st["T"])
    st.update({f"Y{k}": ys[k] for k in range(5)})
    return {k: np.ascontiguousarray(v + np.zeros((nx, ny, nz))) for k, v in st.items()}


SPEEDS = (128, 120, 128)


def speeds(N):
    """SHA-256 of the flame speeds of a sheared flow, in which the flame is wrinkled in one cell of seven."""
    nx, ny, nz = SPEEDS
    i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
    st = state(nx, ny, nz)
    for f, q in (("u", 7 * i + 3 * j + 5 * k), ("v", 5 * i + 11 * j + 2 * k), ("w", 3 * i + 2 * j + 13 * k)):
        st[f] = np.abs(q % 16 - 8.0) / 8.0
    ctx = N.Context(config(nx, ny, nz), precision=N.FP32)
    ctx.upload_attribute(N.initial_state(config(nx, ny, nz))[0])
    ctx.upload_state(st)
    ctx.eval_rhs(0)
    h = hashlib.sha256(ctx.field("ST").astype(np.float32).tobytes()).hexdigest()
    ctx.close()
    return h


def main():
    from lesgpu import native as N
    out = {}
    for name, (nx, ny, nz, start) in CASES.items():
        s = N.Solver(config(nx, ny, nz), precision=N.FP32, start_step=start)
        s.ctx.upload_state(state(nx, ny, nz, name == "ties"))
        s.run(STEPS)
        for f, v in s.state().items():
            out[f"{name}_{f}"] = v.astype(np.float32)
        out[f"{name}_dt"] = np.float64(s.last_dt)
        s.close()
    out["speeds"] = np.array(speeds(N))
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(HERE, "fp32_ref.npz"), **out)


if __name__ == "__main__":
    main()
