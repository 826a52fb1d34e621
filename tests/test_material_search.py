"""The search for a material index in dt/eps grids (material.h), on the host:
compiled into a small library and compared with numpy.  At most 256 triples,
told apart by their bits, signed zeros and NaN payloads included, give an index
and its table; a 257th anywhere gives none; and a structure whose many triples
lie in its middle is given up on early."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oidt_b200.build import HERE

SRC = """
#include "material.h"
template <typename T> static size_t run(const T *x, const T *y, const T *z, size_t nx, size_t plane, uint8_t *idx, T *tab) {
  const T *const cb[3] = {x, y, z};
  std::vector<T> t;
  const size_t seen = oidt::find_mat<T>(cb, nx, plane, idx, t);
  for (size_t q = 0; q < t.size(); ++q) tab[q] = t[q];
  return seen;
}
extern "C" size_t find32(const float *x, const float *y, const float *z, size_t nx, size_t p, uint8_t *i, float *t) {
  return run(x, y, z, nx, p, i, t);
}
extern "C" size_t find64(const double *x, const double *y, const double *z, size_t nx, size_t p, uint8_t *i, double *t) {
  return run(x, y, z, nx, p, i, t);
}
"""


@pytest.fixture(scope="module")
def find(tmp_path_factory):
    d = tmp_path_factory.mktemp("material")
    (d / "m.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(HERE, "csrc"), "-o", str(d / "m.so"),
                    str(d / "m.cpp")], check=True)
    lib = C.CDLL(str(d / "m.so"))

    def run(grids, nx):
        dt = grids[0].dtype
        fn = lib.find32 if dt == np.float32 else lib.find64
        fn.restype = C.c_size_t
        n = grids[0].size
        idx, tab = np.full(n, 255, np.uint8), np.zeros((256, 4), dt)
        seen = fn(*[g.ctypes.data_as(C.c_void_p) for g in grids], C.c_size_t(nx), C.c_size_t(n // nx),
                  idx.ctypes.data_as(C.c_void_p), tab.ctypes.data_as(C.c_void_p))
        return seen, idx, tab
    return run


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nx,plane", [(1, 1), (5, 31), (2, 32), (3, 33), (8, 500), (13, 63), (10, 410), (1, 4099), (4099, 1)])
@pytest.mark.parametrize("triples", [1, 2, 255, 256])
def test_index_and_table(find, dtype, nx, plane, triples):
    n = nx * plane
    rng = np.random.default_rng(n + triples)
    pick = np.repeat(rng.integers(0, triples, n), 1 + rng.integers(0, 80, n))[:n]  # runs about the 32 cells' length
    pick[: min(triples, n)] = np.arange(min(triples, n))
    tabs = [(1.0 + rng.random(triples)).astype(dtype) for _ in range(3)]
    tabs[0][:], tabs[1][:] = tabs[0][0], tabs[1][0]  # told apart by the last one, or by a sign or payload
    if triples > 1:
        tabs[2][0], tabs[2][1] = 0.0, -0.0
    if triples > 2:
        nan = _bits(np.array([np.nan, np.nan], dtype))
        nan[1] += 1
        tabs[2][2:4] = nan.view(dtype)
    grids = [np.ascontiguousarray(t[pick]) for t in tabs]
    seen, idx, tab = find(grids, nx)
    assert seen == n
    assert len(np.unique(idx)) == len(np.unique(pick))
    for k in range(3):
        np.testing.assert_array_equal(_bits(np.ascontiguousarray(tab[idx, k])), _bits(grids[k]))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("where", [0, 585, 2047, 2048, 2051, 2056, 4094])
def test_a_257th_triple_anywhere(find, dtype, where):
    n, nx = 4095, 7
    x = (1.0 + (np.arange(n) % 256)).astype(dtype)
    y, z = np.ones(n, dtype), np.ones(n, dtype)
    assert find([x, y, z], nx)[0] == n
    y[where] = -1.0
    assert find([x, y, z], nx)[0] < n


@pytest.mark.parametrize("at,most", [((24, 40), 0.02), ((0, 7), 0.25), ((57, 64), 0.25), ((40, 47), 0.25)])
def test_many_triples_are_met_early(find, at, most):
    """A core in the middle, at once; one of a tenth of the planes anywhere, in
    a quarter of the pass (steps of 0.618 nx: ten planes leave no gap of 7)."""
    nx, ny, nz = 64, 40, 96
    g = [np.ones((nx, ny, nz), np.float32) for _ in range(3)]
    rng = np.random.default_rng(0)
    g[1][at[0]:at[1], 15:25, 10:-10] = rng.random((at[1] - at[0], 10, nz - 20))
    seen, _, _ = find([np.ascontiguousarray(a.ravel()) for a in g], nx)
    assert seen < nx * ny * nz * most
