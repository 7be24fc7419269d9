"""A batch that has been captured follows a later rc_set_priority of its
members: the next run builds the launches again (seen by the failure armed at
the march's launch, which a plain replay never meets) and the results keep
every bit."""
import numpy as np
import pytest

from radchan_b200 import _lib as L
from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _arm(n):
    L.check(L.lib().rc_debug_fail_next(b"march", n))


def test_captured_batch_follows_set_priority():
    tabs = W.tables_nb(nB=20, nQ=4, nT=16)
    probs = [W.channel_params(12, 10, 8, photmax=12, nVar=2, nB=20, nQ=4, nT=16),
             W.channel_params(8, 6, 10, grey=True, photmax=20, nVar=2)]
    ss = [api.Solver(p, None if p.grey else tabs) for p in probs]
    T = [W.channel_field(p, seed=3) for p in probs]
    ref = [s.solve(t) for s, t in zip(ss, T)]
    b = api.Batch(use_graph=True)
    for s, t in zip(ss, T):
        b.add(s, t)

    def check():
        b.run()
        b.wait()
        for i, r in enumerate(ref):
            np.testing.assert_array_equal(b.collect(i).q64, r.q64)

    try:
        check()
        _arm(1)
        check()            # replayed: no march is launched by the host
        ss[1].set_priority(12.0)  # RC_PRIORITY_DEFAULT, as it is
        check()            # replayed too
        for k, thr in enumerate((0.0, 2.0, 1e6)):
            ss[k % 2].set_priority(thr)
            _arm(1)
            with pytest.raises(L.RadChanError, match="march"):
                b.run()
            check()
            _arm(1)
            check()
    finally:
        _arm(0)
    b.close()
    for s in ss:
        s.close()
