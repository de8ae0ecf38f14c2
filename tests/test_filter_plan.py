"""The form of the R-weighting filter the device runs (tr_filter_host.h,
rweight_plan), on the CPU: where the pad's part is taken from the row's ends
the transform is shorter, and its result is the oracle's."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O

CSRC = Path(__file__).resolve().parents[1] / "autom2_b200" / "csrc"
PROBE = r"""
#include "tr_filter_host.h"
extern "C" int probe_plan(int nx, size_t smem, int *dims, float *ghat, float *ramp) {
  trb::RweightSpectrum s, p;
  const bool ok = trb::rweight_plan(nx, smem, &s);
  if (ok != trb::rweight_spectrum(nx, smem, &p)) return -1;
  if (!ok) return 0;
  dims[0] = s.npad, dims[1] = s.log2m, dims[2] = p.log2m, dims[3] = (int)s.ramp.size();
  for (size_t i = 0; i < s.ghat.size(); ++i) ghat[2 * i] = s.ghat[i].x, ghat[2 * i + 1] = s.ghat[i].y;
  for (size_t i = 0; i < s.ramp.size(); ++i) ramp[2 * i] = s.ramp[i].x, ramp[2 * i + 1] = s.ramp[i].y;
  return 1;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory, cuda_include):
    d = tmp_path_factory.mktemp("planprobe")
    (d / "p.cpp").write_text(PROBE)
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}",
                    f"-I{cuda_include}", str(d / "p.cpp"), "-o", str(d / "p.so")], check=True)
    lib = C.CDLL(str(d / "p.so"))

    def get(nx, smem=200 * 1024):
        dims = (C.c_int * 4)()
        g, r = np.zeros(1 << 16, np.float32), np.zeros(1 << 15, np.float32)
        ok = lib.probe_plan(nx, C.c_size_t(smem), dims, g.ctypes.data_as(C.c_void_p),
                            r.ctypes.data_as(C.c_void_p))
        assert ok >= 0, "the plan refuses other sizes than the padded form"
        if not ok:
            return None
        return list(dims), g[:2 << dims[1]].view(np.complex64).astype(complex), \
            r[:2 * dims[3]].reshape(-1, 2).astype(float)

    return get


@pytest.mark.parametrize("nx,short", [(2, False), (16, False), (61, False), (64, True), (65, False),
                                      (100, False), (256, True), (257, False), (717, False),
                                      (1000, True), (1024, True), (4096, True)])
def test_plan_reproduces_the_reference_filter(plan, nx, short):
    (npad, log2m, padded_log2m, nramp), ghat, ramp = plan(nx)
    assert (nramp == nx) == short and (log2m < padded_log2m) == short
    assert (1 << log2m) >= npad + nx - 1
    rows = np.random.default_rng(nx).normal(size=(4, nx)).astype(np.float32)
    rows[1] += 3.0  # an offset row: the ramp pad matters
    rows[2, -1] += 50.0  # and one with a step at its end
    x = np.zeros((4, ghat.size))
    x[:, :nx] = rows
    if not short:
        j, nxp = np.arange(nx, npad), npad - nx + 1
        x[:, nx:npad] = (j - nx + 1) / nxp * rows[:, :1] + (npad - j) / nxp * rows[:, -1:]
    y = (np.fft.ifft(np.fft.fft(x, axis=1) * ghat, axis=1) * ghat.size)[:, :nx].real
    if short:
        y += ramp[:, 0] * rows[:, :1] + ramp[:, 1] * rows[:, -1:]
    want = O.Restatement().filter_rweight(rows.copy())
    for a, b in zip(y, want):
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 2e-6


def test_refusals_are_the_padded_forms(plan):
    for nx, smem in ((9000, 200 * 1024), (8192, 200 * 1024), (7400, 200 * 1024), (4096, 64 * 1024),
                     (2048, 30 * 1024)):
        plan(nx, smem)  # asserts that both forms refuse, or neither
