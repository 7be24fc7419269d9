"""The source terms' divisions by the coupling's constants, done with a
rounded reciprocal and exact remainders: equal to the plain IEEE divisions of
the oracle for constants and values that are awkward to round, for zero
fluxes (one replicate: sigma 0), for non-finite results, and for constants
outside the range the reciprocal form is used in."""
import numpy as np
import pytest

from oracle import dns as OD
from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu

CONST = [dict(), dict(stefan=float(np.nextafter(2.0, 1.0))), dict(stefan=1.0 / 3.0, Height=float(np.nextafter(1.0, 0.0))),
         dict(Height=-0.7), dict(stefan=-5.67e-8, Height=3.0), dict(stefan=1e-70, Height=1e70), dict(stefan=1e300),
         dict(Height=1e-310)]


@pytest.mark.parametrize("nvar", [1, 3])
@pytest.mark.parametrize("const", range(len(CONST)))
def test_constant_divisions_equal_ieee_division(const, nvar):
    tabs = W.tables_nb(nB=20, nQ=4, nT=16)
    p = W.channel_params(24, 13, 11, photmax=7, nVar=nvar, nB=20, nQ=4, nT=16, calcwalls=1, adiabw=1, adiabe=1)
    T = W.channel_field(p, seed=const)
    a = tabs.arrays()
    cpl = api.DnsCoupling(Tin=873.1, Height=0.37, underrelax=0.7, Tnb=a["Tnb"].astype(np.float64),
                          kP=a["kP"].astype(np.float64))
    for k, v in CONST[const].items():
        setattr(cpl, k, v)
    T1 = T.astype(np.float64) / cpl.Tin
    s = api.Solver(p, tabs)
    r = s.solve(T)
    h = s.dns_source(s.solve_async(T), cpl, T1)
    with np.errstate(all="ignore"):
        want = OD.dns_source(r.Q, r.sigma, T1, cpl.Tin, cpl.Height, cpl.underrelax, cpl.stefan, cpl.Tnb, cpl.kP, 1,
                             p.jmax)
    for k in ("Qnew", "Varnew", "Knew", "Gnew"):
        np.testing.assert_array_equal(h[k], want[k], err_msg=k)
    s.close()
