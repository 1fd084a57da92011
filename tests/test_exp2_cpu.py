"""2^x from an exponent in 64 bits (csrc/exp2_of_double.h), as the host compiles it, against numpy's in extended precision."""
import ctypes
import os
import subprocess

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "enterprise-inference_b200", "csrc")


def test_exp2_of_double(tmp_path):
    src, so = tmp_path / "e.cpp", tmp_path / "e.so"
    src.write_text('#include "exp2_of_double.h"\nextern "C" void f(const double* x, float* y, int n) { for (int i = 0; i < n; ++i) y[i] = b200::exp2_of_double(x[i]); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).f

    def f(x):
        x, y = np.ascontiguousarray(x, dtype=np.float64), np.empty(len(x), dtype=np.float32)
        fn(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), len(x))
        return y

    rng = np.random.default_rng(1)
    x = np.concatenate([-rng.uniform(0, 120, 400000), -rng.uniform(0, 1.5, 400000), -np.arange(0, 120.5, 0.5), -np.exp(rng.uniform(-40, 0, 1000)), [0.0, -0.0, -120.0]])
    want = np.exp2(x.astype(np.longdouble))
    # its last rounding (2^-24 of the result) and what q's roundings leave: q = 0.69 + 0.24 f + .. is half a unit off in its last step (2^-25) and the one before,
    # times |f| <= 1/2 over 2^f >= 0.71: 2^-24.5
    assert (np.abs(f(x).astype(np.longdouble) - want) <= (2.0 ** -24 + 2.0 ** -24.5) * want).all()
    y = f(np.array([-120.0001, -1e9, -np.inf, np.nan]))
    assert (y[:3] == 0).all() and np.isnan(y[3])
