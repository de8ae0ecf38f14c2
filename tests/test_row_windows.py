"""Windows of the row-invariant tiles (tr_geom.h compiled as host C++): which
geometries qualify, and that a tile's voxels never reach a detector column
outside its window, over random tilts and tile positions."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "autom2_b200" / "csrc"
PROBE = r"""
#include "tr_geom.h"
extern "C" int probe_rows(const double *c8, int nt, int *out) {
  static trb::TiltGeo g[256];
  trb::GeomInfo gi;
  int bad = -1;
  const int s = trb::derive_geometry(c8, nt, 1024, 1024, 256, (size_t)1 << 30, g, &gi, &bad);
  out[0] = gi.rows, out[1] = gi.rbp_cols, out[2] = gi.rfp_cols;
  out[3] = trb::kRowBpX, out[4] = trb::kRowBpZ, out[5] = trb::kRowFpX, out[6] = trb::kRowFpZ;
  return s;
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory, cuda_include):
    d = tmp_path_factory.mktemp("rowprobe")
    (d / "p.cpp").write_text(PROBE)
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}",
                    f"-I{cuda_include}", str(d / "p.cpp"), "-o", str(d / "p.so")], check=True)
    lib = C.CDLL(str(d / "p.so"))

    def call(c8):
        c8 = np.ascontiguousarray(c8, np.float64)
        out = (C.c_int * 7)()
        assert lib.probe_rows(c8.ctypes.data_as(C.POINTER(C.c_double)), len(c8), out) == 0
        return list(out)

    return call


def _tilt(deg, b=(0.0, 0.0, 1.0, 0.0), a2=0.0, a1=None):
    t = np.deg2rad(deg)
    return [0.3, np.cos(t) if a1 is None else a1, a2, -np.sin(t), *b]


@pytest.mark.parametrize("tilts,ok", [
    ([_tilt(-60), _tilt(0), _tilt(60)], True),
    ([_tilt(10, b=(4.7, 0.0, 1.0, 0.0))], True),            # a row shift
    ([_tilt(10), _tilt(10, a2=1e-9)], False),               # the column depends on the row
    ([_tilt(10, b=(0.0, 0.0, 1.0, 1e-9))], False),          # the row depends on the section
    ([_tilt(10, b=(0.0, 1e-9, 1.0, 0.0))], False),
    ([_tilt(10, a1=1.0001)], False),                        # more than a column a step
    ([_tilt(100)], False),                                  # a1 < 0
])
def test_which_geometries_qualify(rows, tilts, ok):
    assert bool(rows(tilts)[0]) == ok


def test_windows_hold_every_column_a_tile_reaches(rows):
    rng = np.random.default_rng(5)
    for _ in range(200):
        deg = rng.uniform(-90, 90, rng.integers(1, 6))
        c8 = [_tilt(d) for d in deg]
        ok, bp, fp, bx, bz, fx, fz = rows(c8)
        assert ok
        for cols, ex, ez in ((bp, bx, bz), (fp, fx, fz)):
            x, z = np.meshgrid(np.arange(ex), np.arange(ez))
            for k in c8:
                for u0 in rng.uniform(-50, 50, 8):
                    # 2^-20 px: far above the fixed-point coordinates' error
                    u = u0 + k[1] * x + k[3] * z
                    kmin = np.floor(u.min()) - 1
                    assert np.floor(u.min() - 2.0 ** -20) >= kmin
                    assert np.floor(u.max() + 2.0 ** -20) + 1 < kmin + cols
