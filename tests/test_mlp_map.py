"""The parameter layout of the warm-start MLP (twmc_mlp_map.h) on the CPU: the
BF16 copy's element of every parameter, at the corners of each layer, for the
largest layer that the network accepts among them (65536 x 65536: 2^32
weights)."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pincosimulator_gb300", "csrc")
SOURCE = """
#include "twmc_mlp_map.h"
extern "C" int64_t slot(int nl, const int* widths, int l, int64_t i) {
  twmc::LayerMap m{};
  int64_t off = 0, h = 0;
  for (int j = 0; j < nl; ++j) {
    m.off[j] = off; m.h[j] = h; m.n[j] = widths[j + 1]; m.k[j] = widths[j]; m.ld[j] = (widths[j] + 7) & ~7;
    off += int64_t(m.n[j]) * m.k[j] + m.n[j];
    h += int64_t(m.n[j]) * m.ld[j];
  }
  return twmc::weight_slot(m, l, i);
}
"""


@pytest.fixture(scope="module")
def slot(tmp_path_factory):
    d = tmp_path_factory.mktemp("mlp_map")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "m.cpp"), "-o", str(d / "m.so")], check=True)
    f = C.CDLL(str(d / "m.so")).slot
    f.restype, f.argtypes = C.c_int64, [C.c_int, C.POINTER(C.c_int), C.c_int, C.c_int64]
    return lambda widths, l, i: f(len(widths) - 1, (C.c_int * len(widths))(*widths), l, i)


@pytest.mark.parametrize("widths", [[5, 3], [1, 1, 1], [5, 65536, 65536, 2049], [65536, 65535, 7], [65536, 65536]])
def test_weight_slots(slot, widths):
    off = h = 0
    for l, (k, n) in enumerate(zip(widths[:-1], widths[1:])):
        ld = (k + 7) // 8 * 8
        for r in {0, 1, n // 2, n - 1} & set(range(n)):
            for c in {0, 1, k // 2, k - 1} & set(range(k)):
                assert slot(widths, l, off + r * k + c) == h + r * ld + c
            assert slot(widths, l, off + n * k + r) == -1, "a bias has no place in the weights' copy"
        off += n * k + n
        h += n * ld
