"""Row-invariant geometries (no XTILT, no in-plane rotation) take kernels whose
tiles are 16 x 8 voxels by 128 rows: sizes around those edges, both layouts,
odd and misaligned volumes, windows beyond the stack, against the FP64
oracle.  Tolerance: the parity bar of the FP32 kernels, relative L2 1e-5."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu
TOL = 1e-5

# nx, ny, nt, th, layout, largest tilt, shift sigma; the last two have too few
# tilts for the forward projection's kernel.
CASES = [
    (257, 256, 24, 128, 0, 70, 1.0),
    (250, 127, 25, 130, 1, 85, 2.0),
    (200, 250, 24, 100, 0, 60, 40.0),
    (96, 1025, 24, 35, 1, 89, 300.0),
    (321, 385, 24, 33, 0, 45, 0.3),
    (257, 129, 5, 40, 1, 60, 1.0),
    (272, 128, 1, 57, 0, 50, 0.5),
]


def _case(restatement, nx, ny, nt, th, layout, amax, shift):
    rng = np.random.default_rng(nx * 1000 + ny + nt)
    ang = np.linspace(-amax, amax, nt) if nt > 1 else [amax]
    c8 = restatement.coeffs(np.asarray(ang, np.float32), 0.0, 0.0, 0.0)
    c8[:, 0] += rng.normal(0, 1, nt) * shift
    c8[:, 4] += rng.normal(0, 1, nt) * min(shift, 5.0)
    c8[nt // 2, 4] = 2.0  # a whole-row shift
    proj = rng.normal(size=(nt, ny, nx)).astype(np.float32)
    vol = rng.normal(size=(ny, th, nx) if layout == 0 else (th, ny, nx)).astype(np.float32)
    return c8, proj, vol, T.default_origin(layout, nx, ny, th)


def _misaligned(a):
    """The array on the GPU, its first element 4 bytes past a 16-byte boundary."""
    t = torch.empty(a.size + 1, device="cuda")[1:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("misaligned", [False, True])
@pytest.mark.parametrize("nx,ny,nt,th,layout,amax,shift", CASES)
def test_projections(engine, restatement, nx, ny, nt, th, layout, amax, shift, misaligned):
    R = restatement
    c8, proj, vol, org = _case(R, nx, ny, nt, th, layout, amax, shift)
    put = _misaligned if misaligned else (lambda a: torch.from_numpy(a).cuda())
    g = R.geom(nx, ny, nt, th, layout, 0, org)
    engine.set_problem(nx, ny, nt, th, c8, layout, org)
    v = put(vol)
    engine.backproject(put(proj), v)
    assert O.rel_l2(v.cpu().numpy(), R.backproject(g, c8, proj, vol, fp64=True)) < TOL
    val, wt = torch.zeros((nt, ny, nx), device="cuda"), torch.zeros((nt, ny, nx), device="cuda")
    engine.forward_project(put(vol), val, wt)
    want = [R.reproject(g, c8[t], vol, fp64=True) for t in range(nt)]
    assert O.rel_l2(val.cpu().numpy(), np.stack([w[0] for w in want])) < TOL
    assert O.rel_l2(wt.cpu().numpy(), np.stack([w[1] for w in want])) < TOL


@pytest.mark.parametrize("nx,ny,nt,th,layout,amax,shift", CASES[1:4])
def test_sirt_and_a_slab_of_sections(engine, restatement, nx, ny, nt, th, layout, amax, shift):
    R = restatement
    c8, proj, vol, org = _case(R, nx, ny, nt, th, layout, amax, shift)
    g = R.geom(nx, ny, nt, th, layout, 0, org)
    engine.set_problem(nx, ny, nt, th, c8, layout, org)
    v = torch.from_numpy(vol).cuda()
    engine.sirt(torch.from_numpy(proj).cuda(), v, 2, 0.5)
    want = R.sirt(g, c8, proj, vol, 2, 0.5, fp64=True)
    assert O.rel_l2(v.cpu().numpy(), want) < TOL
    # a stack that 16 bits hold exactly, FP32 residuals: the same iteration
    whole16 = np.round(proj * 8)
    for dtype in (torch.float16, torch.bfloat16):
        q, scale = engine.quantize(torch.from_numpy(whole16).cuda(), dtype)
        v = torch.from_numpy(vol).cuda()
        engine.sirt_lp(q, scale, v, 2, 0.5, "f32")
        assert O.rel_l2(v.cpu().numpy(), R.sirt(g, c8, whole16, vol, 2, 0.5, fp64=True)) < TOL
    # sections [z0, z0 + nz) alone: the same voxels as the whole volume's
    z0, nz = 5, th - 9
    whole = torch.zeros(vol.shape, device="cuda")
    part = torch.zeros_like(whole)
    p = torch.from_numpy(proj).cuda()
    engine.backproject(p, whole)
    first = part[:, z0:] if layout == 0 else part[z0:]
    engine.backproject(p, first, z0, nz)
    cut = (slice(None), slice(z0, z0 + nz)) if layout == 0 else (slice(z0, z0 + nz),)
    assert O.rel_l2(part[cut].cpu().numpy(), whole[cut].cpu().numpy()) < 1e-6
    part[cut] = 0
    assert float(part.abs().max()) == 0.0


@pytest.mark.parametrize("nx,ny,nt,th", [(250, 250, 17, 66), (242, 240, 16, 70),
                                          (256, 128, 33, 96)])
def test_compensated_sums_of_16_bit_stacks(engine, restatement, nx, ny, nt, th):
    """Tilt counts at and beside the groups that are summed plainly.  Plain sums
    of 16 tilts and one rounding of the total stay within 10 x 2**-24 of sums of
    like sign; the values here are positive."""
    R = restatement
    c8, proj, vol, org = _case(R, nx, ny, nt, th, 0, 60, 0.0)
    proj, vol = np.abs(proj), np.abs(vol)
    g = R.geom(nx, ny, nt, th, 0, 0, org)
    engine.set_problem(nx, ny, nt, th, c8, 0, org)
    q, scale = engine.quantize(torch.from_numpy(proj).cuda(), torch.float16)
    exact = (q.float() * scale[:, None, None]).cpu().numpy()
    v = torch.from_numpy(vol).cuda()
    engine.backproject_lp(q, scale, v)
    assert O.rel_l2(v.cpu().numpy(), R.backproject(g, c8, exact, vol, fp64=True)) < 6e-7


def test_two_streams_share_a_context(engine, restatement):
    """Back-projections queued on two streams without a synchronisation between
    them each see their own stack."""
    R = restatement
    nx, ny, nt, th, layout, amax, shift = CASES[5]
    c8, proj, vol, org = _case(R, nx, ny, nt, th, layout, amax, shift)
    engine.set_problem(nx, ny, nt, th, c8, layout, org)
    p = [torch.from_numpy(proj).cuda() * s for s in (1.0, -3.0)]
    v = [torch.zeros(vol.shape, device="cuda") for _ in p]
    streams = [torch.cuda.Stream() for _ in p]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, a, b in zip(streams, p, v):
            with torch.cuda.stream(s):
                b.zero_()
                engine.backproject(a, b)
    torch.cuda.synchronize()
    want = R.backproject(R.geom(nx, ny, nt, th, layout, 0, org), c8, proj, 0 * vol, fp64=True)
    for b, s in zip(v, (1.0, -3.0)):
        assert O.rel_l2(b.cpu().numpy(), s * want) < TOL


def test_an_infinite_edge_pixel_stays_inside_the_image(engine, restatement):
    """Voxels that no pixel reaches get nothing, also beside a pixel that is not
    finite, and voxels between it and its neighbour are not finite."""
    R = restatement
    nx, ny, nt, th = 256, 128, 3, 64
    c8 = R.coeffs(np.array([-40, 0.5, 30], np.float32), 0.0, 0.0, 0.0)
    proj = np.random.default_rng(3).normal(size=(nt, ny, nx)).astype(np.float32)
    proj[0, 5, 0] = np.inf
    proj[2, 9, nx - 1] = -np.inf
    org = T.default_origin(0, nx, ny, th)
    engine.set_problem(nx, ny, nt, th, c8, T.LAYOUT_Y, org)
    v = torch.zeros((ny, th, nx), device="cuda")
    engine.backproject(torch.from_numpy(proj).cuda(), v)
    want = R.backproject(R.geom(nx, ny, nt, th, 0, 0, org), c8, proj, np.zeros((ny, th, nx)),
                         fp64=True)
    got = v.cpu().numpy()
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert O.rel_l2(got[ok], want[ok]) < TOL
