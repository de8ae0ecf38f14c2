"""The memory a context holds between calls."""
import numpy as np
import pytest
import torch

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
