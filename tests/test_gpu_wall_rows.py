"""The rows of a wall whose flux is not computed are 0 in every result, also in
memory that another solve has used: the solve itself writes them."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu

N = (12, 9, 7)


def _params(west, east, **kw):
    return W.channel_params(*N, grey=True, photmax=8, nVar=2, calcwalls=int(west or east), adiabw=west, adiabe=east, **kw)


def _check(p, qw, vw, what):
    for w, on in ((0, p.adiabw), (1, p.adiabe)):
        for a in (qw, vw):
            assert np.any(a[w] != 0) if on else np.all(a[w] == 0), (what, w)


@pytest.mark.parametrize("fp64", [0, 1])
def test_rows_of_walls_without_a_flux_are_zero(fp64):
    used = [api.Solver(_params(1, 1, floatpoint=fp64)) for _ in range(4)]
    T = W.channel_field(used[0].p, seed=1)
    for _ in range(2):
        for s in used:
            t = [s.solve_async(T), s.solve_async(T)]
            for x in t:
                s.collect(x)
    for s in used:
        s.close()  # its memory, full of wall fluxes, goes to the next contexts
    for west, east in ((0, 0), (1, 0), (0, 1)):
        p = _params(west, east, floatpoint=fp64)
        s = api.Solver(p)
        for _ in range(3):
            r = s.solve(T)
            _check(p, r.qw64, r.vw64, "solve")
        b = api.Batch()
        b.add(s, T)
        for _ in range(2):
            b.run()
            b.wait()
            r = b.collect(0)
            _check(p, r.qw64, r.vw64, "batch")
            np.testing.assert_array_equal(r.Q[1:-1, 1:-1, 0] != 0, np.full((N[2], N[1]), bool(west)))
        b.close()
        s.close()
