"""ADMM on row-invariant geometries, whose normalised projection is formed between
the row stacks, against the deterministic mode, which takes the general kernels:
both layouts, sizes beside the tiles', 128-row blocks that are partly empty, shifts
that leave detector rows and columns without a weight.  Tolerance: the parity bar of
the FP32 kernels, relative L2 1e-5."""
import numpy as np
import pytest
import torch

import oracle as O
from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nt,th,layout,shift", [
    (257, 256, 24, 128, 0, 0.0),
    (250, 127, 25, 130, 1, 2.0),
    (200, 250, 24, 100, 0, 30.0),
])
def test_admm(engine, restatement, nx, ny, nt, th, layout, shift):
    rng = np.random.default_rng(nx)
    c8 = restatement.coeffs(np.linspace(-60, 60, nt).astype(np.float32), 0.0, 0.0, 0.0)
    c8[:, 0] += rng.normal(0, 1, nt) * shift
    c8[:, 4] += rng.normal(0, 1, nt) * min(shift, 4.0)
    proj = torch.from_numpy(rng.normal(size=(nt, ny, nx)).astype(np.float32)).cuda()
    shape = (ny, th, nx) if layout == 0 else (th, ny, nx)
    got = []
    for exact in (False, True):
        engine.set_problem(nx, ny, nt, th, c8, layout, T.default_origin(layout, nx, ny, th))
        engine.set_deterministic(exact)
        v = torch.zeros(shape, device="cuda")
        engine.admm(proj, v, 2, 1, 0.5, 0.02)
        engine.set_deterministic(False)
        got.append(v.cpu().numpy())
    assert O.rel_l2(got[0], got[1]) < 1e-5
