"""The device memory a scheduler holds: within its budget while uneven jobs follow
one another, and given back when it has been idle."""
import threading
import time

import numpy as np
import pytest
import torch

from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu

SLACK = 64 << 20  # the step tables and spectra, and the pool's rounding of each buffer


def test_jobs_and_kept_memory_stay_within_the_budget():
    """Series whose buffers grow from one to the next, so that none fits what the
    one before gave back."""
    nx, ny, th = 256, 512, 32
    tilts = [31, 73, 131, 211, 307, 401]
    c8 = {nt: T.geometry_from_angles(np.linspace(-60, 60, nt).astype(np.float32)) for nt in tilts}
    stacks = {nt: torch.randn((nt, ny, nx), device="cuda") for nt in tilts}
    vols = {nt: torch.zeros((ny, th, nx), device="cuda") for nt in tilts}
    budget = 2 * tilts[-1] * ny * nx * 4 + (64 << 20)  # the largest job's two stacks and weights
    s = T.Scheduler(0, hbm_budget=budget)
    try:
        torch.cuda.synchronize()
        base = torch.cuda.mem_get_info()[0]
        least, stop = [base], threading.Event()

        def watch():
            while not stop.is_set():
                least[0] = min(least[0], torch.cuda.mem_get_info()[0])

        w = threading.Thread(target=watch)
        w.start()
        for _ in range(2):
            ids = [s.submit(s.job(stacks[nt], vols[nt], c8[nt], 0, wbp=True, sirt_iters=1))
                   for nt in tilts]
            for i in ids:
                s.wait(i)
        stop.set()
        w.join()
        assert base - least[0] <= budget + SLACK
        end = time.time() + 10
        while base - torch.cuda.mem_get_info()[0] > SLACK and time.time() < end:
            time.sleep(0.1)
        assert base - torch.cuda.mem_get_info()[0] <= SLACK
    finally:
        s.close()
