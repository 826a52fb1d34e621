"""The kappa dx tables as a job uploads them (kappa.h, compiled for the host):
the values, their correctly rounded reciprocals, and 1 in the padding, so that
a group of the vector form that reaches into it stays in the fast quotient's
range (reciprocals of 2^-20 to 2^50 in float32, 2^-100 to 2^100 in float64)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oidt_b200.build import HERE

SRC = """
#include "kappa.h"
template <typename T> static void run(const T *kd, size_t n, size_t padded, T *k, T *r) {
  std::vector<T> a, b(3, T(7));
  oidt::kappa_rows<T>(kd, n, padded, a, b);
  for (size_t i = 0; i < padded; ++i) k[i] = a[i], r[i] = b[i];
}
extern "C" void rows32(const float *kd, size_t n, size_t p, float *k, float *r) { run(kd, n, p, k, r); }
extern "C" void rows64(const double *kd, size_t n, size_t p, double *k, double *r) { run(kd, n, p, k, r); }
"""


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_padding_is_in_range(tmp_path, dtype):
    (tmp_path / "k.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(HERE, "csrc"), "-o",
                    str(tmp_path / "k.so"), str(tmp_path / "k.cpp")], check=True)
    lib = C.CDLL(str(tmp_path / "k.so"))
    fn = lib.rows32 if dtype == np.float32 else lib.rows64
    rng = np.random.default_rng(1)
    lo, hi = (2.0 ** -20, 2.0 ** 50) if dtype == np.float32 else (2.0 ** -100, 2.0 ** 100)
    for n in range(5, 13):
        p = -(-n // 4) * 4
        kd = (2e-8 * (1 + 4 * rng.random(n))).astype(dtype)
        k, r = np.full(p, 9, dtype), np.full(p, 9, dtype)
        fn(*[C.c_void_p(kd.ctypes.data), C.c_size_t(n), C.c_size_t(p), C.c_void_p(k.ctypes.data), C.c_void_p(r.ctypes.data)])
        np.testing.assert_array_equal(k[:n], kd)
        np.testing.assert_array_equal(r[:n], dtype(1) / kd)
        np.testing.assert_array_equal(k[n:], 1)
        np.testing.assert_array_equal(r[n:], 1)
        assert np.all((r >= lo) & (r <= hi))
