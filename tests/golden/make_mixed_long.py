"""Writes tests/golden/mixed_long.npz: long simulations and their gradients on mixed contexts (CUDA
library, default transform paths), 100 steps at rho = 10.

FP32 transforms leave rounding of 6e-8 of a field's maximum everywhere, and the logistic reaction
multiplies it by up to exp(rho T) = 2e4 here. So these results follow every rounding of a solve's
transforms: a path that computes the same in another order of operations moves the final states by 5e-5 to 8e-3. The
inputs are exact in FP32 (dyadic numbers from integer voxel indices), so that they are the same on
every machine.

    python tests/golden/make_mixed_long.py
"""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, ROOT)

OUT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "mixed_long.npz")
SIZES = (24, 32, 64)  # cuFFT's transforms at the first two, the library's own passes at 64
NT, RHO, KAPPA = 100, 10.0, 0.0125


def compute(n):
    from glia_gb300 import _abi, native
    from glia_gb300.context import Context

    i = np.arange(n)
    x, y, z = i[:, None, None], i[None, :, None], i[None, None, :]

    def r2(a, b, c):
        return (x - a) ** 2 + (y - b) ** 2 + (z - c) ** 2

    def smooth(f):  # binomial, twice along each axis
        f = f.astype(np.float64)
        for axis in (0, 0, 1, 1, 2, 2):
            f = (np.roll(f, 1, axis) + 2 * f + np.roll(f, -1, axis)) / 4
        return f

    h = n // 2
    brain = r2(h, h, h) < (3 * n // 8) ** 2
    white = brain & ((x // 8 + y // 8 + z // 8) % 2 == 0)
    ctx = Context(native.load(), n, _abi.GLIA_MIXED)
    ctx.set_time(0.01, NT)
    ctx.set_tissue(*(smooth(m).reshape(-1) for m in (white, brain & ~white, ~brain)))
    ctx.set_coefficients(k=KAPPA, rho=RHO, k_gm_wm=0.25)
    c0 = (np.maximum(0.0, 1.0 - r2(h, h + 2, h - 1) / 16.0) ** 2 / 2).reshape(-1)
    c1 = ctx.solve_state(c0).reshape((n,) * 3)[:: n // 24, :: n // 24, :: n // 24]
    v = 2 * np.pi / n
    centers = v * np.array([[h, h, h], [h + 3, h, h], [h, h - 3, h + 2], [h - 2, h + 1, h]]) + 0.01
    ctx.set_phi(centers, 1.5 * v, 1.0)
    ctx.set_opt(np=4, nk=1, nr=1, diffusivity_inversion=0, beta=0.0, all_gradients=1)
    ctx.set_history(_abi.GLIA_HISTORY_CHECKPOINT, 10)
    d1 = (r2(h - 1, h, h + 1) < (n // 4) ** 2).astype(np.float64).reshape(-1)
    J, dJ = ctx.eval_objective_and_gradient(
        np.array([0.5, 0.0, 0.25, 0.0, KAPPA, RHO]), d1)
    ctx.close()
    return np.ascontiguousarray(c1, dtype=np.float32), np.concatenate([[J], dJ])


if __name__ == "__main__":
    out = {}
    for n in SIZES:
        out[f"c1_{n}"], out[f"gradient_{n}"] = compute(n)
    np.savez_compressed(OUT, **out)
    print({k: (v.shape, float(np.linalg.norm(v))) for k, v in out.items()})
