"""Projection weights of separable geometries as a column's times a row's,
against the oracle's FP64 splat of ones: sections of a volume, a subset of the
tilts, shifts beyond the image, steep tilts on both sides of the rule (|a1| >=
0.05), added to what the caller holds.  Tolerance: relative L2 1e-5, the parity
bar of the FP32 kernels."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,th,layout,angles,shift", [
    (33, 7, 5, 0, [0.0], 0.0),
    (64, 300, 40, 1, [-60, -13, 0, 31, 75], 1.0),
    (100, 20, 64, 0, [-86, 86.5, 10], 3.0),      # |a1| 0.07
    (50, 9, 30, 0, [-89.5, 20], 0.5),            # a steeper tilt: the splat
    (40, 31, 12, 1, [-30, 45], 60.0),            # mostly outside the image
])
def test_weights(engine, restatement, nx, ny, th, layout, angles, shift):
    R = restatement
    rng = np.random.default_rng(nx)
    nt = len(angles)
    c8 = R.coeffs(np.asarray(angles, np.float32), 0.0, 0.0, 0.0)
    c8[:, 0] += rng.normal(0, 1, nt) * shift
    c8[:, 4] += rng.normal(0, 1, nt) * shift
    c8[0, 4] = np.round(c8[0, 4])  # whole rows
    org = T.default_origin(layout, nx, ny, th)
    engine.set_problem(nx, ny, nt, th, c8, layout, org)
    vol = torch.zeros((ny, th, nx) if layout == 0 else (th, ny, nx), device="cuda")

    def want(t, z0, nz):
        g = R.geom(nx, ny, 1, nz, layout, z0, org)
        ones = np.ones((ny, nz, nx) if layout == 0 else (nz, ny, nx))
        return R.reproject(g, c8[t], ones, fp64=True)[1]

    val, wt = torch.zeros((nt, ny, nx), device="cuda"), torch.full((nt, ny, nx), 2.0, device="cuda")
    engine.forward_project(vol, val, wt)
    ref = np.stack([want(t, 0, th) for t in range(nt)])
    assert O.rel_l2(wt.cpu().numpy() - 2.0, ref) < 1e-5
    if th > 8:
        z0, nz, t0 = 3, th - 5, nt - 1
        first = vol[:, z0:] if layout == 0 else vol[z0:]
        v1, w1 = torch.zeros((1, ny, nx), device="cuda"), torch.zeros((1, ny, nx), device="cuda")
        engine.forward_project_tilts(first, t0, 1, v1, w1, z0, nz)
        assert O.rel_l2(w1.cpu().numpy()[0], want(t0, z0, nz)) < 1e-5
