"""What a handle keeps between calls, and the copies of large results."""
import dataclasses

import numpy as np
import pytest
import torch

from adga_b200 import Ladder, synth

pytestmark = pytest.mark.gpu

KEPT = 32 * 2 ** 20        # the bound on a handle's work buffer


def ladder(nk, iwf):
    return Ladder.from_problem(synth.make_problem(
        dataclasses.replace(synth.SPECS["t2"], name="w2", nk=(nk,) * 3, nq=(1, 1, 1), iwf=iwf, iwb=0), quick_mu=True))


def test_large_work_buffers_are_given_back():
    """post_loop on 32^3 k-points works on 4 x 2 x 24 x 32768 numbers (101 MB)."""
    small, lad = ladder(4, 4), ladder(32, 24)
    try:
        small.post_loop(want=("n_dga",))      # loads the kernels and their local memory
        before = torch.cuda.mem_get_info()[0]
        lad.post_loop(want=("n_dga",))
        held = before - torch.cuda.mem_get_info()[0]
    finally:
        small.close()
        lad.close()
    assert held <= KEPT + 16 * 2 ** 20        # and what the driver rounds up
