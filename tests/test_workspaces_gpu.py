"""What a handle keeps between calls, and the copies of large results."""
import dataclasses

import numpy as np
import pytest
import torch

from adga_b200 import Ladder, synth
from tests.helpers import library_env, rel_err

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


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_batches_stay_within_the_grid(prec):
    """A 32^3 q mesh (32768 points, 65536 matrices) of one orbital would fit the
    memory as one batch; the same results as from batches of 5000 points."""
    p = synth.make_problem(dataclasses.replace(synth.SPECS["t1"], name="w1", nk=(32,) * 3, nq=(32,) * 3, iwf=41,
                                               iwb=0), quick_mu=True)
    out = []
    for settings in ({}, {"ADGA_BATCH": "5000"}):
        with library_env(settings):
            lad = Ladder.from_problem(p)
            try:
                lad.set_vertex(0, *p.vertex(0))
                status, stats = lad.ladder_run(1, None, prec)
                assert not status.any() and stats["points"] == 32768
                out.append({k: np.array(v) for k, v in lad.get_outputs().items()})
            finally:
                lad.close()
    for k in ("chi_qw_dens", "chi_qw_magn", "sigma_nl"):
        assert rel_err(out[0][k], out[1][k]) < (1e-12 if prec == "fp64" else 1e-9), k


def test_large_results_into_pageable_memory():
    """42 x 8000 numbers (5.4 MB, ten chunks of 512 KB and a part of one) go into
    pageable memory through the driver for the handle's first 256 MB and through
    four threads' staging after, directly into page-locked: the same bytes, each
    time others, with fresh and reused arrays."""
    p = synth.make_problem(dataclasses.replace(synth.SPECS["t1"], name="w3", nk=(20,) * 3, nq=(2,) * 3, iwf=21,
                                               iwb=0), quick_mu=True)
    lad = Ladder.from_problem(p)
    try:
        lad.set_vertex(0, *p.vertex(0))
        lad.ladder_run(1, None, "fp64")
        pinned = {k: torch.zeros(tuple(reversed(v)), dtype=torch.complex128, pin_memory=True).numpy().T
                  for k, v in lad.output_shapes(8).items()}
        reused = {k: np.zeros(v, complex, order="F") for k, v in lad.output_shapes(8).items()}
        last = None
        for _ in range(40):                           # 2 x 40 copies, 430 MB
            lad.ladder_run(1, None, "fp64")           # the sums go on: another self-energy each time
            want = lad.get_outputs(pinned)["sigma_nl"]
            assert want.nbytes == 5376000 and np.abs(want).min() > 0
            assert last is None or not np.array_equal(want, last)
            last = want.copy()
            assert np.array_equal(lad.get_outputs()["sigma_nl"], last)
            assert np.array_equal(lad.get_outputs(reused)["sigma_nl"], last)
    finally:
        lad.close()
