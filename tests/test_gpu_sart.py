"""SART's sweeps (the update of one tilt and the projection at the next in one
pass) against the FP64 oracle: general and separable geometries, odd and
misaligned volumes, both layouts, windows across the image border, one tilt.
Tolerance: the parity bar of the FP32 kernels, relative L2 1e-5."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("misaligned", [False, True])
@pytest.mark.parametrize("nx,ny,nt,th,layout,pitch,rot,shift,iters", [
    (64, 4, 3, 32, 0, 0.0, 0.0, 0.0, 1),
    (65, 9, 5, 33, 1, 0.0, 0.0, 3.0, 2),
    (129, 31, 4, 40, 0, 4.0, 2.0, 1.0, 2),
    (200, 50, 6, 17, 1, 0.3, 0.5, 20.0, 1),
    (70, 12, 1, 20, 0, 0.0, 1.0, 0.0, 3),
])
def test_sart(engine, restatement, nx, ny, nt, th, layout, pitch, rot, shift, iters, misaligned):
    R = restatement
    rng = np.random.default_rng(nx + ny)
    c8 = R.coeffs(np.linspace(-55, 60, nt).astype(np.float32), 0.0, pitch, 0.0)
    psi = np.deg2rad(rng.normal(0, rot, nt))[:, None]
    if rot:
        a, b = c8[:, :4].copy(), c8[:, 4:].copy()
        c8[:, :4], c8[:, 4:] = np.cos(psi) * a - np.sin(psi) * b, np.sin(psi) * a + np.cos(psi) * b
    c8[:, 0] += rng.normal(0, 1, nt) * shift
    c8[:, 4] += rng.normal(0, 1, nt) * min(shift, 3.0)
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = rng.normal(size=(ny, th, nx) if layout == 0 else (th, ny, nx)).astype(np.float32)
    org = T.default_origin(layout, nx, ny, th)
    engine.set_problem(nx, ny, nt, th, c8, layout, org)
    v = torch.empty(vol.size + 1, device="cuda")[int(misaligned):][:vol.size].view(vol.shape)
    v.copy_(torch.from_numpy(vol))
    engine.sart(torch.from_numpy(proj).cuda(), v, iters, 0.4)
    want = R.sart(R.geom(nx, ny, nt, th, layout, 0, org), c8, proj, vol, iters, 0.4, fp64=True)
    assert O.rel_l2(v.cpu().numpy(), want) < 1e-5


def test_sart_whole_pixel_shifts(engine, restatement):
    """Shifts of whole pixels put voxel rows exactly a pixel above the image,
    where no tap has a weight: they get nothing.  Tolerance as above."""
    R = restatement
    rng = np.random.default_rng(3)
    nx, ny, nt, th = 66, 12, 3, 20
    c8 = R.coeffs(np.linspace(-40, 45, nt).astype(np.float32), 0.0, 0.0, 0.0)
    c8[:, 4] += [-3.0, -1.0, 2.0]
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = np.zeros((ny, th, nx), np.float32)
    org = T.default_origin(0, nx, ny, th)
    engine.set_problem(nx, ny, nt, th, c8, 0, org)
    v = torch.from_numpy(vol.copy()).cuda()
    engine.sart(torch.from_numpy(proj).cuda(), v, 1, 0.4)
    want = R.sart(R.geom(nx, ny, nt, th, 0, 0, org), c8, proj, vol, 1, 0.4, fp64=True)
    assert O.rel_l2(v.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("scale", [2.2, 2.4])
def test_sart_wide_windows(engine, restatement, scale):
    """A rotated, magnified detector: windows whose two tables just fit a sweep's
    shared memory, and ones that take separate projections.  Tolerance as above."""
    R = restatement
    rng = np.random.default_rng(5)
    nx, ny, nt, th = 70, 40, 3, 34
    c8 = R.coeffs(np.linspace(-50, 50, nt).astype(np.float32), 0.0, 0.0, 0.0)
    a, b = c8[:, :4].copy(), c8[:, 4:].copy()
    c8[:, :4], c8[:, 4:] = (a - b) * np.sqrt(0.5) * scale, (a + b) * np.sqrt(0.5) * scale
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = rng.normal(size=(ny, th, nx)).astype(np.float32)
    org = T.default_origin(0, nx, ny, th)
    engine.set_problem(nx, ny, nt, th, c8, 0, org)
    v = torch.from_numpy(vol.copy()).cuda()
    engine.sart(torch.from_numpy(proj).cuda(), v, 2, 0.4)
    want = R.sart(R.geom(nx, ny, nt, th, 0, 0, org), c8, proj, vol, 2, 0.4, fp64=True)
    assert O.rel_l2(v.cpu().numpy(), want) < 1e-5
