"""Row-invariant projections of more tilts than one launch takes, in groups that are
even and uneven, against the deterministic mode, which takes the general kernel.
Tolerance: the parity bar of the FP32 kernels, relative L2 1e-5."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,shear", [(150, 0), (151, 0), (181, 0), (301, 0), (455, 0),
                                      (40, 1), (40, 0.9)])
def test_projections_of_many_tilts(engine, nt, shear):
    """shear: the section's step of every tilt, with a column's of one (windows wider
    than a rotation's); 0: rotations."""
    nx, ny, th = 250, 250, 130
    rng = np.random.default_rng(nt)
    c8 = T.geometry_from_angles(np.linspace(-70, 70, nt).astype(np.float32)).copy()
    if shear:
        c8[:, 1], c8[:, 3] = 1.0, shear
    c8[:, 0] += rng.normal(0, 2, nt)
    c8[:, 4] += rng.normal(0, 2, nt)
    vol = torch.randn((ny, th, nx), device="cuda")
    proj = torch.randn((nt, ny, nx), device="cuda")
    engine.set_problem(nx, ny, nt, th, c8, T.LAYOUT_Y)
    got = []
    for exact in (False, True):
        engine.set_deterministic(exact)
        val, v = torch.ones((nt, ny, nx), device="cuda"), vol.clone()
        engine.forward_project(vol, val)
        engine.sirt(proj, v, 1, 0.5)
        engine.set_deterministic(False)
        got.append((val.cpu().numpy(), v.cpu().numpy()))
    for a, b in zip(*got):
        assert O.rel_l2(a, b) < 1e-5
