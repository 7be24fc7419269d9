"""The source terms' index arithmetic: the 32-bit kernel up to its limit (cells
of the padded pencil times the longer edge below 4e9) and the 64-bit one from
there on, with either edge the longer; and the table row's division for steps
whose truncation is 1 K, that fit 16 bits and that do not.  All outputs are
those of the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import dns as OD
from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu

TIN = 955.0


def _run(n, Tnb, T1=None, jstart=1, jend=-1):
    p = W.channel_params(*n, grey=True, photmax=2, nVar=2, calcwalls=1, adiabw=1, adiabe=1)
    p.abscoeff = 4000.0
    T = W.channel_field(p, seed=6)
    rng = np.random.default_rng(5)
    kP = rng.uniform(0.1, 2.0, len(Tnb))
    cpl = api.DnsCoupling(Tin=TIN, Height=0.5, underrelax=0.8, Tnb=Tnb, kP=kP, jstart=jstart, jend=jend)
    if T1 is None:
        T1 = T.astype(np.float64) / TIN
    je = p.jmax if jend < 0 else jend
    T1 = np.ascontiguousarray(T1[:, jstart - 1:je + 2, :])
    s = api.Solver(p)
    r = s.solve(T)
    h = s.dns_source(s.solve_async(T), cpl, T1)
    s.close()
    want = OD.dns_source(r.Q, r.sigma, T1, cpl.Tin, cpl.Height, cpl.underrelax, cpl.stefan, cpl.Tnb, cpl.kP, jstart, je)
    for k in ("Qnew", "Varnew", "Knew", "Gnew"):
        np.testing.assert_array_equal(h[k], want[k], err_msg=k)
    assert h["n_clamped"] == want["n_clamped"]


def _is_small(n, jn):
    return float(n[0] + 2) * max(n[1], jn + 2) * (n[2] + 2) * max(n[0] + 2, jn) < 4.0e9


@pytest.mark.parametrize("n,small", [((4000, 10, 18), True), ((4000, 10, 19), False), ((4, 4000, 39), True),
                                     ((4, 4000, 40), False)])
def test_both_index_widths_equal_the_oracle(n, small):
    assert _is_small(n, n[1]) == small
    _run(n, np.linspace(400.0, 1300.0, 64))


def test_part_of_the_rows_in_64_bits():
    assert not _is_small((4000, 16, 19), 9)
    _run((4000, 16, 19), np.linspace(400.0, 1300.0, 64), jstart=5, jend=13)


@pytest.mark.parametrize("step,rows", [(1.0, 120), (1.5, 120), (1.999, 120), (2.0, 120), (65535.5, 3), (65536.0, 3),
                                       (3.0e6, 4)])
def test_row_divisions_equal_the_oracle(step, rows):
    n = (12, 9, 7)
    T0 = 700.0
    rng = np.random.default_rng(7)
    # temperatures before, in and past the table, on its rows and between
    x = T0 + step * rng.uniform(-2, rows + 2, (n[2] + 2, n[1] + 2, n[0] + 2))
    on = rng.random(x.shape) < 0.3
    x[on] = T0 + step * rng.integers(-2, rows + 2, x.shape)[on]
    _run(n, T0 + step * np.arange(rows), T1=x / TIN)
