"""The collision's arithmetic on the host against the oracle, over the whole
range of the limiter (infinite: none)."""
import ctypes as C
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def collide(tmp_path_factory):
    out = tmp_path_factory.mktemp("collide") / "collide_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-x", "c++",
                    str(ROOT / "tests" / "drivers" / "collide_check.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.collide_check_f32.argtypes = [C.c_void_p, C.c_int, C.c_float, C.c_float]
    lib.collide_check_f64.argtypes = [C.c_void_p, C.c_int, C.c_double, C.c_double]

    def run(f, nu, limiter):
        f = f.copy()
        fn = lib.collide_check_f64 if f.dtype == np.float64 else lib.collide_check_f32
        fn(f.ctypes.data, f.shape[1], nu, limiter)
        return f
    return run


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("limiter", [1e-39, 0.05, 1e10, 1e31, 1e38, 3.4028234e38, math.inf])
def test_limiter_range(collide, dtype, limiter):
    """Tolerance: about ten roundings of single-precision values, relative to
    the largest population."""
    rng = np.random.default_rng(11)
    f = np.stack([O.feq(*rng.uniform(-0.06, 0.06, 4)) for _ in range(40)], axis=1)
    f = (f * (1 + 0.05 * rng.standard_normal(f.shape))).astype(np.float32)
    ref = O.apply_collision_batch(f, nu=0.02, limiter=limiter)
    got = collide(f.astype(dtype), 0.02, limiter)
    assert np.max(np.abs(got - ref)) / np.abs(ref).max() < 2e-6
