"""Results collected in any order and form, two solves in flight: floats only,
everything, device copies.  Blocks up to 2 MB come back through a staging block
that the first collect asking for doubles pins, larger ones straight into the
caller's arrays; both sides of that size."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(9, 7, 5), (43, 43, 45), (48, 46, 44)])
def test_collect_forms_agree_in_any_order(n):
    p = W.channel_params(*n, grey=True, photmax=4, nVar=2, calcwalls=1, adiabw=1, adiabe=1)
    T = [W.channel_field(p, seed=i) for i in range(2)]
    ref = []
    for t in T:
        s = api.Solver(p)
        ref.append(s.solve(t))
        s.close()

    def floats(i, tk):
        Q, S = (np.zeros(api.result_shape(p), np.float32) for _ in range(2))
        s.collect_into(tk, Q, S)
        np.testing.assert_array_equal(Q, ref[i].Q)
        np.testing.assert_array_equal(S, ref[i].sigma)

    def everything(i, tk):
        r = s.collect(tk)
        for k in ("Q", "sigma", "q64", "var64", "qw64", "vw64"):
            np.testing.assert_array_equal(getattr(r, k), getattr(ref[i], k), err_msg=k)

    s = api.Solver(p)
    for order in ((floats, floats), (floats, everything), (everything, floats), (everything, everything)):
        for first in (0, 1):
            tk = [s.solve_async(t) for t in T]
            order[0](first, tk[first])
            order[1](1 - first, tk[1 - first])
    s.close()
