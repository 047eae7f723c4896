"""Long mixed simulations give the answers they always gave (tests/golden/mixed_long.npz, made by
tests/golden/make_mixed_long.py): every FP32 solve keeps the transforms, and so the rounding, that
the reaction then amplifies by exp(rho T).

Tolerances: float results are held to 2e-5 of their norm, and at any value to 8e-4 of the larger
of that value and the root mean square. Equal roundings give equal bits; another order of operations
inside the solves moves the final states by 5e-5 to 8e-3, at single voxels by 2e-3 to 0.2."""
import os

import numpy as np
import pytest

from tests.golden.make_mixed_long import SIZES, compute

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_long.npz")


def far(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    rms = np.linalg.norm(b) / np.sqrt(b.size)
    return (np.linalg.norm(a - b) / np.linalg.norm(b),
            np.max(np.abs(a - b) / np.maximum(rms, np.abs(b))))


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_long_mixed_results_stay(n):
    golden = np.load(GOLDEN)
    for name, got in zip(("c1", "gradient"), compute(n)):
        rel, single = far(got, golden[f"{name}_{n}"])
        assert rel <= 2e-5 and single <= 8e-4, (name, rel, single)
