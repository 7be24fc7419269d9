"""Grids with one very long axis: every cell index up to the limit of the
packed cell (65535 an axis) and across the sign bit of its half word, bit for
bit against the oracle.  The gas is thick, so that paths stay short."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2, 40000, 2), (2, 65535, 1), (2, 2, 65535), (65535, 2, 1)])
def test_long_axis_equals_the_oracle(n):
    from oracle import oracle as O
    p = W.channel_params(*n, grey=True, photmax=2, nVar=1, calcwalls=1, adiabw=1, adiabe=1)
    p.abscoeff = 2000.0
    T = W.channel_field(p, seed=2)
    s = api.Solver(p)
    r = s.solve(T)
    o = O.solve(p, None, T, rpt=s.get_launch()[0])
    np.testing.assert_array_equal(r.q64, o["q64"])
    np.testing.assert_array_equal(r.qw64, o["qw64"])
    s.close()
