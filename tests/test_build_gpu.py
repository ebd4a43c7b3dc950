"""The BSE build's kernels (one orbital; two and three without V(q); four, five
and V(q) on the FP64 tensor cores) through one solved point, at orbital counts,
boxes and tiles with remainders: eta and gamma^q_d against the oracle."""
import dataclasses

import numpy as np
import pytest

from adga_b200 import Ladder, synth
from oracle.adga_oracle import Oracle, read_vq_transform
from tests.helpers import rel_err, to_inputs

pytestmark = pytest.mark.gpu


def make(ndim, iwf):
    base = synth.SPECS[{1: "t1", 2: "t2", 3: "t3"}.get(ndim, "t5")]
    return synth.make_problem(dataclasses.replace(base, name=f"b{ndim}", ndim=ndim, iwf=iwf, offdiag=0.03))


@pytest.mark.parametrize("ndim,iwf", [(1, 1), (1, 17), (2, 1), (2, 9), (3, 2), (3, 5), (4, 1), (4, 3), (5, 1), (5, 3)])
@pytest.mark.parametrize("with_vq", [False, True])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("mixed", 1e-8)])
def test_point_matches_oracle(ndim, iwf, with_vq, prec, tol):
    p = make(ndim, iwf)
    s = p.spec
    inp = to_inputs(p)
    lad = Ladder.from_problem(p)
    try:
        if with_vq:
            rng = np.random.default_rng(ndim)
            shape = (ndim,) * 4 + (s.nqp,)
            vq = 0.1 * (rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape))
            lad.set_vq(vq)
            inp.vq = read_vq_transform(vq)
        lad.set_vertex(1, *p.vertex(1))
        iq = min(2, s.nqp)
        ed, em, gq, info = lad.bse_point(iq, 1, prec)
    finally:
        lad.close()
    o = Oracle(inp)
    out = dict(bubble_loc=np.zeros((s.ndim2, s.ndim2, 2 * s.iwb + 1), complex),
               chi_loc_dens=np.zeros((s.ndim2, s.ndim2, 2 * s.iwb + 1), complex),
               chi_loc_magn=np.zeros((s.ndim2, s.ndim2, 2 * s.iwb + 1), complex))
    want = o.point(iq - 1, 1, o.local_block(1, iq - 1, out))
    assert info == 0
    for got, key in ((ed, "etaqd"), (em, "etaqm"), (gq, "gammaqd")):
        assert rel_err(got, want[key]) < tol, (key, rel_err(got, want[key]))


@pytest.mark.parametrize("iwf", [31, 32, 33, 48, 63, 65])
def test_unpivoted_blocks_match_oracle(iwf):
    """The unpivoted FP32 block LU of 64 columns at full and partial last blocks
    (N = 62 .. 130: 62, 64, 2, 32, 62 and 2 columns), with the refinement's
    tolerance of 1e-10 on the residual, condition numbers below 100."""
    test_point_matches_oracle(1, iwf, False, "mixed", 1e-8)
