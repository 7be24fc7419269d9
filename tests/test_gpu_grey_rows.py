"""Grey tables of more than 256 rows.  Cells hold their table coordinate in 16
bits with 8 fraction bits: as long as the field's hottest cell lies below row
256 of the table (which ends 10% above it) the solve is the oracle's, and
beyond that row it is reported instead of answered."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(rows, **kw):
    p = W.channel_params(10, 8, 6, grey=True, photmax=16, nVar=2, calcwalls=1, adiabw=1, adiabe=1, **kw)
    p.grey_nT = rows
    return p, W.channel_field(p, seed=4)


@pytest.mark.parametrize("rows", [256, 257, 290])
def test_hot_cells_below_row_256_equal_the_oracle(rows):
    from oracle import oracle as O
    p, T = _problem(rows)
    s = api.Solver(p)
    r = s.solve(T)
    o = O.solve(p, None, T, rpt=s.get_launch()[0])
    np.testing.assert_array_equal(r.q64, o["q64"])
    np.testing.assert_array_equal(r.qw64, o["qw64"])
    s.close()


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("bd_y", [1, 3])
def test_hot_cells_beyond_row_256_are_reported(bd_y, fp64):
    p, T = _problem(360, bd_y=bd_y, floatpoint=fp64)
    s = api.Solver(p)
    for _ in range(2):  # the context goes on
        t = s.solve_async(T)
        assert s.info(t).status & 16
        with pytest.raises(Exception, match="grey_nT"):
            s.collect(t)
    s.close()
    b = api.Batch()
    s = api.Solver(p)
    b.add(s, T)
    b.run()
    b.wait()
    with pytest.raises(Exception, match="grey_nT"):
        b.collect(0)
    b.close()
    s.close()
