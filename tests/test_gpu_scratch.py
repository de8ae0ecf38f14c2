"""The memory a context holds between calls."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


def _tilts(nt, shift=0.3):
    c8 = T.geometry_from_angles(np.linspace(-60, 60, nt).astype(np.float32)).copy()
    c8[:, 0] += shift
    return c8


def test_scratch_that_no_problem_claims_is_given_back():
    """ADMM's seven volumes stay for three problems that do not use them and are
    gone at the fourth."""
    nx, ny, nt, th = 64, 32, 5, 40
    admm = 7 * nx * ny * th * 4
    e = T.Engine(0)
    try:
        p = torch.randn((nt, ny, nx), device="cuda")
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        e.admm(p, torch.zeros((ny, th, nx), device="cuda"), 1, 1, 0.5, 0.02)
        assert e.scratch_bytes > admm
        for k in range(4):
            e.set_problem(nx, ny, nt, th, _tilts(nt))
            e.sirt(p, torch.zeros((ny, th, nx), device="cuda"), 1, 0.5)
            assert (e.scratch_bytes > admm) == (k < 3)
        # and come back for a problem that does
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        e.admm(p, torch.zeros((ny, th, nx), device="cuda"), 1, 1, 0.5, 0.02)
        assert e.scratch_bytes > admm
    finally:
        e.close()


def test_a_row_stack_holds_the_launch_s_tilts_only():
    """SART back-projects single tilts of a row-invariant geometry: beside its
    stacks (and the int64 sums of the deterministic mode) a context holds one
    tilt's row stack at most, not one that grows to the whole series'.  Both modes
    agree to the parity bar of the FP32 kernels, relative L2 1e-5."""
    nx, ny, nt, th = 1024, 512, 6, 64
    p = torch.randn((nt, ny, nx), device="cuda")
    got = []
    for deterministic in (False, True):
        e = T.Engine(0)
        try:
            e.set_problem(nx, ny, nt, th, _tilts(nt))
            e.set_deterministic(deterministic)
            v = torch.zeros((ny, th, nx), device="cuda")
            e.sart(p, v, 1, 0.3)
            torch.cuda.synchronize()
            stacks = nt * ny * nx * 4 * (4 if deterministic else 2)
            tilt = ny * (nx + 2 * 64) * 4  # windows are less than 64 columns wide
            assert e.scratch_bytes <= stacks + tilt + 4096
            got.append(v)
        finally:
            e.close()
    assert O.rel_l2(got[0].cpu().numpy(), got[1].cpu().numpy()) < 1e-5


def test_a_projection_beside_a_capture():
    """Projections on a stream of their own, on a context that has no scratch yet,
    leave the capture of another stream as it is."""
    nx, ny, nt, th = 512, 256, 41, 64
    p = torch.randn((nt, ny, nx), device="cuda")
    v = torch.zeros((ny, th, nx), device="cuda")
    val = torch.zeros_like(p)
    x = torch.zeros(8, device="cuda")
    side = torch.cuda.Stream()
    e = T.Engine(0)
    try:
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            x += 1
            with torch.cuda.stream(side):
                e.backproject(p, v)
                e.forward_project(v, val)
        graph.replay()
        torch.cuda.synchronize()
        assert e.scratch_bytes > 0  # the row stacks
        assert float(x.min()) == float(x.max()) == 1.0
        again = torch.zeros_like(v)
        e.backproject(p, again)
        assert torch.equal(v, again)
    finally:
        e.close()


def test_deterministic_results_do_not_depend_on_the_scratch():
    """The same back-projection, with room for a row stack and with none."""
    nx, ny, nt, th = 512, 256, 41, 64
    p = torch.randn((nt, ny, nx), device="cuda")
    got = []
    for budget in (0, 1):
        e = T.Engine(0, hbm_budget=budget)
        try:
            e.set_problem(nx, ny, nt, th, _tilts(nt))
            e.set_deterministic(True)
            v = torch.zeros((ny, th, nx), device="cuda")
            e.backproject(p, v)
            got.append(v)
        finally:
            e.close()
    assert torch.equal(*got)


@pytest.mark.parametrize("room", [0, 1, 2])
def test_sirt_with_room_for_some_of_the_row_stacks(room):
    """Budgets that hold SIRT's own scratch and none, one or both of the row stacks
    (the projection's and the back-projection's): the same volume, to the parity bar
    of the FP32 kernels, and a budget that is kept."""
    nx, ny, nt, th = 512, 256, 41, 64
    p = torch.randn((nt, ny, nx), device="cuda")
    stack = nt * ny * nx * 4
    want = torch.zeros((ny, th, nx), device="cuda")
    e = T.Engine(0)
    try:
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        e.set_deterministic(True)
        e.sirt(p, want, 2, 0.5)
        # without the int64 sums and the largest magnitude of the deterministic mode
        need = e.scratch_bytes - 2 * stack - 4
    finally:
        e.close()
    e = T.Engine(0, hbm_budget=need + room * (stack * 5 // 4) + 4096)
    try:
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        v = torch.zeros_like(want)
        e.sirt(p, v, 2, 0.5)
        torch.cuda.synchronize()
        assert e.scratch_bytes <= need + room * (stack * 5 // 4) + 4096
        assert e.scratch_bytes >= need + room * stack
        assert O.rel_l2(v.cpu().numpy(), want.cpu().numpy()) < 1e-5
    finally:
        e.close()


def test_sirt_under_capture():
    """A captured SIRT call takes kernels that need no row stacks (which the context
    may drop later) and allocates nothing; its replays equal the eager call to the
    parity bar of the FP32 kernels."""
    nx, ny, nt, th = 512, 256, 41, 64
    p = torch.randn((nt, ny, nx), device="cuda")
    e = T.Engine(0)
    try:
        e.set_problem(nx, ny, nt, th, _tilts(nt))
        want = torch.zeros((ny, th, nx), device="cuda")
        e.sirt(p, want, 2, 0.5)
        held = e.scratch_bytes
        v = torch.zeros_like(want)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            e.sirt(p, v, 2, 0.5)
        assert e.scratch_bytes == held
        for _ in range(2):
            v.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert O.rel_l2(v.cpu().numpy(), want.cpu().numpy()) < 1e-5
    finally:
        e.close()
