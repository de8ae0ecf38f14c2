"""Origins (tr_geom.h compiled as host C++): which keep the row-invariant kernels,
and that for those a voxel row's detector row is where the kernels' shared-memory
tiles expect it; origins that leave the int range are refused."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from autom2_b200 import tiltrec as T

CSRC = Path(__file__).resolve().parents[1] / "autom2_b200" / "csrc"
PROBE = r"""
#include "tr_geom.h"
extern "C" int probe(const double *c8, int nt, int nx, int ny, int th, const float *o, int *out) {
  static trb::TiltGeo g[256];
  trb::GeomInfo gi;
  int bad = -1;
  int s = trb::derive_geometry(c8, nt, nx, ny, th, (size_t)1 << 30, g, &gi, &bad);
  if (s == trb::GEOM_OK) s = trb::check_origin(c8, nt, nx, ny, th, o[0], o[1], o[2], &gi, &bad);
  out[0] = gi.rows, out[1] = gi.product_weights, out[2] = trb::GEOM_RANGE;
  return s;
}
"""
NX, NY, TH = 1000, 262140, 200  # the most rows a problem may have


@pytest.fixture(scope="module")
def probe(tmp_path_factory, cuda_include):
    d = tmp_path_factory.mktemp("originprobe")
    (d / "p.cpp").write_text(PROBE)
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}",
                    f"-I{cuda_include}", str(d / "p.cpp"), "-o", str(d / "p.so")], check=True)
    lib = C.CDLL(str(d / "p.so"))

    def call(origin, ny=NY, shift=0.0):
        c8 = T.geometry_from_angles(np.array([-60, 0, 45], np.float32)).copy()
        c8[:, 4] += shift
        out = (C.c_int * 3)()
        s = lib.probe(c8.ctypes.data_as(C.POINTER(C.c_double)), len(c8), NX, ny, TH,
                      (C.c_float * 3)(*origin), out)
        return s, out[0], out[1], out[2]

    return call


def _detector_rows(oy, b0):
    """Lower detector row of every voxel row as the kernels form it, minus the row
    and floor(b0)."""
    y = np.arange(NY)
    off = (y.astype(np.float32) - np.float32(oy)).astype(np.float64)
    return np.floor(b0 + off + float(np.float32(oy))) - y - np.floor(b0)


@pytest.mark.parametrize("oy", [0.0, 511.5, 131070.3, -100.7, 262144.0, -262144.0, 2.6e5 + 0.3])
def test_rows_that_keep_the_kernels_are_where_their_tiles_are(probe, oy):
    s, rows, product, _ = probe((500.0, oy, 100.0))
    assert (s, rows, product) == (0, 1, 1)
    for b0 in (0.0, 0.3, -2.0, 1e-9, -1e-9, 17.999):
        assert np.abs(_detector_rows(oy, b0)).max() <= 1


@pytest.mark.parametrize("oy", [3.0e7, 1.0e8, -9.0e8])
def test_rows_that_would_leave_the_tiles_take_the_general_kernels(probe, oy):
    assert max(np.abs(_detector_rows(oy, b0)).max() for b0 in (0.3, 17.999)) >= 1
    s, rows, product, _ = probe((500.0, oy, 100.0))
    assert (s, rows, product) == (0, 0, 0)


@pytest.mark.parametrize("i", [0, 1, 2])
def test_any_axis_counts(probe, i):
    o = [500.0, 100.0, 100.0]
    o[i] = 3.0e5
    assert probe(o)[:3] == (0, 0, 0)


@pytest.mark.parametrize("origin", [(np.nan, 0, 0), (0, np.inf, 0), (0, 0, -np.inf), (1e12, 0, 0),
                                    (0, 0, 4e9), (3e38, 3e38, 3e38)])
def test_origins_beyond_the_int_range_are_refused(probe, origin):
    s, _, _, refused = probe(origin)
    assert s == refused != 0


@pytest.mark.gpu
def test_refused_by_the_entry_points(engine):
    import torch
    c8 = T.geometry_from_angles(np.array([-60, 0, 45], np.float32))
    p = torch.zeros((3, 8, 16), device="cuda")
    v = torch.zeros((8, 4, 16), device="cuda")
    for origin in ((float("nan"), 4.0, 2.0), (1e12, 4.0, 2.0)):
        with pytest.raises(T.TiltRecError) as e:
            engine.set_problem(16, 8, 3, 4, c8, 0, origin)
        assert e.value.status == -7  # TR_ERR_UNSUPPORTED
        s = T.Scheduler(0)
        try:
            with pytest.raises(T.TiltRecError) as e:
                s.submit(s.job(p, v, c8, 0, origin=origin, wbp=True))
            assert e.value.status == -7
        finally:
            s.close()


@pytest.mark.gpu
def test_a_far_origin_against_the_oracle(engine, restatement):
    """Beyond the row-invariant kernels' origins, rows rounded to two pixels: the
    general kernels, at a size that would take the others.  Tolerance: the parity bar
    of the FP32 kernels, relative L2 1e-5."""
    import torch

    import oracle as O
    R = restatement
    nx, ny, nt, th = 256, 256, 24, 64
    origin = (128.0, 3.0e7, 32.0)
    rng = np.random.default_rng(4)
    c8 = R.coeffs(np.linspace(-50, 50, nt).astype(np.float32), 0.0, 0.0, 0.0)
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = rng.normal(size=(ny, th, nx)).astype(np.float32)
    g = R.geom(nx, ny, nt, th, 0, 0, origin)
    engine.set_problem(nx, ny, nt, th, c8, 0, origin)
    v = torch.from_numpy(vol.copy()).cuda()
    engine.backproject(torch.from_numpy(proj).cuda(), v)
    assert O.rel_l2(v.cpu().numpy(), R.backproject(g, c8, proj, vol, fp64=True)) < 1e-5
    val = torch.zeros((nt, ny, nx), device="cuda")
    engine.forward_project(torch.from_numpy(vol).cuda(), val)
    want = np.stack([R.reproject(g, c8[t], vol, fp64=True)[0] for t in range(nt)])
    assert O.rel_l2(val.cpu().numpy(), want) < 1e-5
