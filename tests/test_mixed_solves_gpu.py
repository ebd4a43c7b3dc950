"""The solves of the mixed path with the FP32 factors, seen apart from the
refinement that corrects them."""
import dataclasses

import numpy as np
import pytest

from adga_b200 import Ladder, synth
from tests.helpers import library_env, oracle_run, rel_err

pytestmark = pytest.mark.gpu


def run(p, settings):
    with library_env(settings):
        lad = Ladder.from_problem(p)
    try:
        for iwb in range(-p.spec.iwb, p.spec.iwb + 1):
            lad.set_vertex(iwb, *p.vertex(iwb))
        status, stats = lad.ladder_run(1, None, "mixed")
        assert not status.any() and stats["mixed_fallbacks"] == 0
        return {k: np.array(v) for k, v in lad.get_outputs().items()}, stats
    finally:
        lad.close()


@pytest.mark.parametrize("iwf", [2, 7, 13])
def test_solves_of_25_right_hand_sides_stay_fp32(iwf):
    """More right-hand sides than the tensor-core solves' 16 (its split keeps
    fewer bits) take the FP32 sums whatever the choice: the same bits."""
    p = synth.make_problem(dataclasses.replace(synth.SPECS["t5"], iwf=iwf))
    default, streaming = run(p, {})[0], run(p, {"ADGA_TRSV_STREAM": "1"})[0]
    for k, v in default.items():
        assert np.array_equal(v, streaming[k]), k


@pytest.mark.parametrize("ndim,iwf", [(1, 31), (1, 32), (1, 33), (1, 48), (1, 63), (1, 65), (2, 8), (2, 9), (3, 4), (3, 7),
                                      (4, 1), (4, 3), (5, 1), (5, 3)])
def test_refinement_corrects_and_does_not_replace(ndim, iwf):
    """Full and partial last blocks of the unpivoted FP32 factorisation (N = 32 to
    150), one to 25 right-hand sides: the oracle's results by at most three
    corrections, no point solved again in FP64 (which would hide a wrong
    factor).  Tolerance of the refinement 1e-10, condition numbers below 100."""
    base = synth.SPECS[{1: "t1", 2: "t2", 3: "t3"}.get(ndim, "t5")]
    p = synth.make_problem(dataclasses.replace(base, name=f"m{ndim}", ndim=ndim, iwf=iwf, iwb=0, offdiag=0.03))
    got, stats = run(p, {})
    want = oracle_run(p)
    assert stats["max_refine_iters"] <= 3
    for k in ("chi_qw_dens", "chi_qw_magn", "sigma_nl"):
        assert rel_err(got[k], want[k]) < 1e-8, (k, rel_err(got[k], want[k]))


@pytest.mark.parametrize("ndim,iwf", [(1, 31), (1, 544), (2, 9), (2, 136), (3, 7), (3, 60), (4, 3), (4, 34)])
def test_first_solve_is_as_good_as_streaming(ndim, iwf):
    """The first correction is the first solve's error.  Both kinds of solve use
    the same FP32 factors, whose error dominates (products of 2^-21 against
    factors of N 2^-24), up to the largest order the tensor-core solves take
    (1088): within a factor of two of each other."""
    base = synth.SPECS[{1: "t1", 2: "t2", 3: "t3"}.get(ndim, "t5")]
    p = synth.make_problem(dataclasses.replace(base, name=f"f{ndim}", ndim=ndim, iwf=iwf, iwb=0, nk=(4,) * 3, nq=(4,) * 3,
                                               offdiag=0.03), quick_mu=True)
    first = []
    for settings in ({}, {"ADGA_TRSV_STREAM": "1"}):
        with library_env({"ADGA_MAX_REFINE": "1", **settings}):
            lad = Ladder.from_problem(p)
        try:
            lad.set_vertex(0, *p.vertex(0))
            first.append(lad.ladder_run(1, None, "mixed")[1]["max_refine_resid"])
        finally:
            lad.close()
    assert 0 < first[0] <= 2 * first[1] and first[1] <= 2 * first[0]


@pytest.mark.parametrize("name", ["t1", "t2", "t3m", "t5"])
@pytest.mark.parametrize("exact", ["0", "1"])
def test_points_without_finite_factors_are_solved_in_fp64(name, exact):
    """A vertex beyond FP32's range leaves the FP32 factors without a finite entry:
    no correction is small beside them, and every point is solved again in FP64,
    to a FP64 run's results (same inputs, tolerance for another batch's sums)."""
    p = synth.make_problem(name)
    npts = p.spec.nqp * (2 * p.spec.iwb + 1)
    outs = []
    for precision in ("mixed", "fp64"):
        with library_env({"ADGA_REFINE_EXACT": exact}):
            lad = Ladder.from_problem(p)
        try:
            for iwb in range(-p.spec.iwb, p.spec.iwb + 1):
                lad.set_vertex(iwb, *(1e40 * np.asarray(v) for v in p.vertex(iwb)))
            status, stats = lad.ladder_run(1, None, precision)
            outs.append({k: np.array(v) for k, v in lad.get_outputs().items()})
        finally:
            lad.close()
        assert stats["mixed_fallbacks"] == (npts if precision == "mixed" else 0)
        assert (status == (-1 if precision == "mixed" else 0)).all()
    for k in ("chi_qw_dens", "chi_qw_magn", "sigma_nl"):
        assert np.isfinite(outs[0][k]).all(), k
        assert rel_err(outs[0][k], outs[1][k]) < 1e-10, k
