"""The vector form's step kernels read their parameter block (about 1 KB) from
kernel parameter space.  A block passed by value, and then by reference to a
function that is not inlined, is first copied into each thread's local memory:
the kernel's stack frame is then larger than the block.  Without the copy a
frame holds spills only (at most 168 bytes a thread as these kernels compile),
so half a block separates the two.  nvcc cross-compiles: no GPU."""
import os
import re
import shutil
import subprocess

import pytest

from oidt_b200.build import FLAGS, HERE, NVCC, ROOT

SRC = """
#include "oidt.h"
#include "kernels.cuh"
#include "vec3d.cuh"
using namespace oidt;
template <typename T, bool X, bool S> void *e() { return (void *)k_v3_e<T, X, S>; }
template <typename T, bool X> void *h() { return (void *)k_v3_h<T, X>; }
template <typename T, bool X, bool S> void *w() { return (void *)k_v3_wave<T, X, S>; }
template <typename T, bool X> struct Forms {  // S: a 'TM' source that the E CPML terms read
  void *f[5] = {e<T, X, kSrcCells<T, X>>(), e<T, X, true>(), h<T, X>(), w<T, X, kSrcCells<T, X>>(), w<T, X, true>()};
};
Forms<float, false> ff;
Forms<float, true> fx;
Forms<double, false> df;
Forms<double, true> dx;
static_assert(sizeof(Params<float>) >= 512 && sizeof(Params<double>) >= 512, "a frame below 512 bytes holds no copy");
"""

TILE = """
#include "oidt.h"
#include "kernels.cuh"
#include "tile2d.cuh"
using namespace oidt;
template <typename T, bool X, int M> void *t() { return (void *)k_2d_tile<T, X, M>; }
void *forms[] = {t<double, false, OIDT_MODE_TM2>(), t<double, false, OIDT_MODE_TE2>(), t<double, true, OIDT_MODE_TM2>(),
                 t<double, true, OIDT_MODE_TE2>(), t<float, true, OIDT_MODE_TM2>(), t<float, true, OIDT_MODE_TE2>()};
"""

pytestmark = pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which(NVCC)), reason="needs nvcc")


def _frames(tmp_path, source, kernel):
    """{kernel instance: bytes of its stack frame}, as the build compiles it."""
    src = tmp_path / "frames.cu"
    src.write_text(source)
    flags = [f for f in FLAGS if f not in ("-shared", "-lineinfo")]
    r = subprocess.run([NVCC] + flags + ["-Xptxas=-v", "-cubin", "-I", os.path.join(HERE, "csrc"), "-I",
                                         os.path.join(ROOT, "include"), "-o", str(tmp_path / "frames.cubin"), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return dict(re.findall(r"Function properties for (\w*%s\w+)\s+(\d+) bytes stack frame" % kernel, r.stderr))


def test_step_kernels_hold_no_copy_of_their_parameters(tmp_path):
    frames = _frames(tmp_path, SRC, "k_v3_")
    assert len(frames) == 18  # float32 EXACT has one instance of each for both
    assert {k: v for k, v in frames.items() if int(v) >= 512} == {}


def test_tile_kernels_keep_a_cell_in_registers(tmp_path):
    """The 2D tile form holds a cell's values and constants in a thread's 64
    registers through the steps.  Spilled there (64 bytes and more a thread),
    float64 fast runs took up to 1.2 times as long; 16 bytes at most spill as
    the kernels compile."""
    frames = _frames(tmp_path, TILE, "k_2d_tile")
    assert len(frames) == 6
    assert {k: v for k, v in frames.items() if int(v) > 32} == {}
