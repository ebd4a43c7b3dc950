"""The solves of the mixed path with the FP32 factors, seen apart from the
refinement that corrects them."""
import dataclasses

import numpy as np
import pytest

from adga_b200 import Ladder, synth
from tests.helpers import library_env

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
