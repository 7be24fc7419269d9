"""A batch that has been captured follows a later rc_set_priority of its
members: the next run builds the launches again (seen by the failure armed at
the march's launch, which a plain replay never meets) and the results keep
every bit.  A list that finds no memory is left out: it is an order only."""
import numpy as np
import pytest

from radchan_b200 import _lib as L
from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _arm(n, site=b"march"):
    L.check(L.lib().rc_debug_fail_next(site, n))


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


def test_no_memory_for_the_list_is_no_failure():
    # more tiles than the march has warps: below that there is no list
    p = W.channel_params(32, 24, 20, grey=True, photmax=40, nVar=2)
    T = W.channel_field(p, seed=3)
    s = api.Solver(p)
    ref = s.solve(T)
    s.close()
    try:
        s = api.Solver(p)
        _arm(1, b"list")
        for _ in range(2):  # without the list, then with it
            np.testing.assert_array_equal(s.solve(T).q64, ref.q64)
        for graph in (False, True):
            b = api.Batch(use_graph=graph)
            x = api.Solver(p)
            b.add(x, T)
            _arm(1, b"list")
            for _ in range(2):
                b.run()
                b.wait()
                np.testing.assert_array_equal(b.collect(0).q64, ref.q64)
            b.close()
            x.close()
        s.close()
    finally:
        _arm(0, b"list")


@pytest.mark.parametrize("graph", [False, True])
def test_first_run_equals_later_runs(graph):
    """The first run of a captured batch goes out before its capture; more
    members than side streams, one of them without a list."""
    ps = [W.channel_params(6 + i % 5, 5, 4 + i % 3, grey=True, photmax=6 + i, nVar=2, seed=i) for i in range(19)]
    ss = [api.Solver(p) for p in ps]
    T = [W.channel_field(p, seed=9) for p in ps]
    ss[3].set_priority(0.0)
    ref = [s.solve(t) for s, t in zip(ss, T)]
    b = api.Batch(use_graph=graph)
    for s, t in zip(ss, T):
        b.add(s, t)
    for _ in range(3):
        b.run()
        assert b.wait() > 0
        assert all(ms >= 0 for ms in b.phases())
        for i, r in enumerate(ref):
            Q, S = (np.zeros(api.result_shape(ps[i]), np.float32) for _ in range(2))
            b.collect_into(i, Q, S)
            np.testing.assert_array_equal(Q, r.Q)
            np.testing.assert_array_equal(b.collect(i).var64, r.var64)
    b.close()
    for s in ss:
        s.close()
