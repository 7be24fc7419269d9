"""Tiles of the long-ray list's first part, marched alone by their warp while
there are no more of them than warps, and with the others beyond that: none, a
few, about as many as warps, and nearly every tile of a near-transparent gas.
Results and steps are the oracle's."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0.05, 0.002])
def test_any_number_of_tiles_marched_alone(k):
    from oracle import oracle as O
    # 8192 tiles of 128 bundles: about twice the warps the GPU holds
    p = W.channel_params(16, 16, 16, grey=True, photmax=64, nVar=4, maxs=[300], calcwalls=1, adiabw=1)
    p.abscoeff = k
    T = W.channel_field(p, seed=8)
    s = api.Solver(p)
    o = O.solve(p, None, T, rpt=s.get_launch()[0])
    for thr in (0.0, 12.0, 1.0, 0.3, 0.1, 0.06, 0.01):
        s.set_priority(thr)
        t = s.solve_async(T)
        steps = s.info(t).steps
        r = s.collect(t)
        np.testing.assert_array_equal(r.q64, o["q64"], err_msg="threshold %g" % thr)
        np.testing.assert_array_equal(r.qw64, o["qw64"])
        assert steps == o["steps"]
    s.close()
