"""Which kernels single projections of row-invariant geometries take (a context
holds a row stack after its first call by the row-invariant ones, and nothing after
the general one), and what the row-invariant ones give at the edges of that choice:
few tilts of thin volumes, two streams, pixels that are not finite.  Tolerance: the
parity bar of the FP32 kernels against the FP64 oracle, relative L2 1e-5."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.fixture
def fresh():
    e = T.Engine(0)
    yield e
    e.close()


def _case(R, nx, ny, nt, th, layout=0):
    rng = np.random.default_rng(nx + ny + nt + th)
    ang = np.linspace(-60, 55, nt) if nt > 1 else [33.0]
    c8 = R.coeffs(np.asarray(ang, np.float32), 0.0, 0.0, 0.0)
    c8[:, 0] += rng.normal(0, 2, nt)
    c8[:, 4] += rng.normal(0, 2, nt)
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = rng.normal(size=(ny, th, nx) if layout == 0 else (th, ny, nx)).astype(np.float32)
    org = T.default_origin(layout, nx, ny, th)
    return c8, proj, vol, org, R.geom(nx, ny, nt, th, layout, 0, org)


@pytest.mark.parametrize("nx,ny,nt,th,layout,rows", [
    (1000, 512, 1, 1, 0, True),
    (1001, 512, 2, 7, 1, True),
    (640, 512, 3, 6, 0, True),
    (250, 250, 24, 66, 0, True),
    (250, 384, 1, 64, 0, False),
    (272, 128, 1, 57, 0, False),
    (512, 256, 8, 32, 1, False),
])
def test_back_projection(fresh, restatement, nx, ny, nt, th, layout, rows):
    R = restatement
    c8, proj, vol, org, g = _case(R, nx, ny, nt, th, layout)
    fresh.set_problem(nx, ny, nt, th, c8, layout, org)
    v = torch.from_numpy(vol.copy()).cuda()
    fresh.backproject(torch.from_numpy(proj).cuda(), v)
    assert (fresh.scratch_bytes > 0) == rows
    assert O.rel_l2(v.cpu().numpy(), R.backproject(g, c8, proj, vol, fp64=True)) < TOL


@pytest.mark.parametrize("nx,ny,nt,th,rows", [
    (250, 512, 41, 28, True),
    (257, 256, 24, 97, True),
    (1000, 330, 24, 32, False),
    (512, 360, 24, 28, False),
])
def test_forward_projection(fresh, restatement, nx, ny, nt, th, rows):
    R = restatement
    c8, _, vol, org, g = _case(R, nx, ny, nt, th)
    fresh.set_problem(nx, ny, nt, th, c8, 0, org)
    val = torch.zeros((nt, ny, nx), device="cuda")
    fresh.forward_project(torch.from_numpy(vol).cuda(), val)
    assert (fresh.scratch_bytes > 0) == rows
    want = np.stack([R.reproject(g, c8[t], vol, fp64=True)[0] for t in range(nt)])
    assert O.rel_l2(val.cpu().numpy(), want) < TOL


def test_two_streams_share_the_row_stacks(fresh, restatement):
    """Projections queued on two streams without a synchronisation between them."""
    R = restatement
    nx, ny, nt, th = 250, 256, 24, 66
    c8, proj, vol, org, g = _case(R, nx, ny, nt, th)
    fresh.set_problem(nx, ny, nt, th, c8, 0, org)
    p = [torch.from_numpy(proj).cuda() * k for k in (1.0, -3.0)]
    w = [torch.from_numpy(vol).cuda() * k for k in (1.0, -3.0)]
    v = [torch.zeros(vol.shape, device="cuda") for _ in p]
    val = [torch.zeros_like(a) for a in p]
    streams = [torch.cuda.Stream() for _ in p]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, a, b, c, d in zip(streams, p, v, w, val):
            with torch.cuda.stream(s):
                b.zero_()
                d.zero_()
                fresh.backproject(a, b)
                fresh.forward_project(c, d)
    torch.cuda.synchronize()
    assert fresh.scratch_bytes > 0
    want_v = R.backproject(g, c8, proj, 0 * vol, fp64=True)
    want_p = np.stack([R.reproject(g, c8[t], vol, fp64=True)[0] for t in range(nt)])
    for b, d, k in zip(v, val, (1.0, -3.0)):
        assert O.rel_l2(b.cpu().numpy(), k * want_v) < TOL
        assert O.rel_l2(d.cpu().numpy(), k * want_p) < TOL


def test_pixels_that_are_not_finite_stay_where_they_reach(fresh, restatement):
    R = restatement
    nx, ny, nt, th = 512, 256, 24, 64
    c8, proj, vol, org, g = _case(R, nx, ny, nt, th)
    proj[0, 5, 0] = np.inf
    proj[12, 9, nx - 1] = -np.inf
    proj[20, 200, 300] = np.nan
    fresh.set_problem(nx, ny, nt, th, c8, 0, org)
    v = torch.zeros(vol.shape, device="cuda")
    fresh.backproject(torch.from_numpy(proj).cuda(), v)
    assert fresh.scratch_bytes > 0
    want = R.backproject(g, c8, proj, 0 * vol, fp64=True)
    got = v.cpu().numpy()
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert O.rel_l2(got[ok], want[ok]) < TOL


@pytest.mark.parametrize("nt", [31, 32, 33])
def test_compensated_sums_at_the_groups_of_tilts(fresh, restatement, nt):
    """As of any stack that 16 bits held: plain sums of 16 tilts and one rounding of
    the total stay within 10 x 2**-24 of sums of like sign."""
    R = restatement
    nx, ny, th = 250, 250, 66
    c8, proj, vol, org, g = _case(R, nx, ny, nt, th)
    c8[:, 0] -= c8[:, 0].mean()
    proj, vol = np.abs(proj), np.abs(vol)
    fresh.set_problem(nx, ny, nt, th, c8, 0, org)
    q, scale = fresh.quantize(torch.from_numpy(proj).cuda(), torch.float16)
    held = fresh.scratch_bytes
    exact = (q.float() * scale[:, None, None]).cpu().numpy()
    v = torch.from_numpy(vol.copy()).cuda()
    fresh.backproject_lp(q, scale, v)
    assert fresh.scratch_bytes > held
    assert O.rel_l2(v.cpu().numpy(), R.backproject(g, c8, exact, vol, fp64=True)) < 6e-7


@pytest.mark.parametrize("resid", ["f32", "f16"])
@pytest.mark.parametrize("layout,depth", [(0, 32), (1, 64), (0, 96)])
def test_slabs_of_sections(fresh, restatement, layout, depth, resid):
    """z-slab SIRT where single projections and whole volumes take the row-invariant
    kernels.  FP32 residuals to the parity bar; FP16 ones keep 11 bits of each pixel's
    residual, of which a voxel averages 41: to 1e-4."""
    R = restatement
    nx, ny, nt, th = 250, 256, 41, 96
    c8, proj, vol, org, g = _case(R, nx, ny, nt, th, layout)
    want = R.sirt(g, c8, proj, vol, 2, 0.5, fp64=True)
    fresh.set_problem(nx, ny, nt, th, c8, layout, org)
    p = torch.from_numpy(proj).cuda()
    for v in (torch.from_numpy(vol.copy()).cuda(), torch.from_numpy(vol.copy()).pin_memory()):
        fresh.sirt_zslabs(p, v, 2, 0.5, depth, resid_dtype=resid)
        torch.cuda.synchronize()
        assert O.rel_l2(v.cpu().numpy(), want) < (TOL if resid == "f32" else 1e-4)
