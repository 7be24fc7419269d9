"""The march's tile bookkeeping and cell entry at the sizes where they can go
wrong, bit for bit against the oracle: tiles that hold one (cell, replicate)
or several, whose items carry over the replicate, row and plane ends; padded
items; the last, partly filled tile and tiles that straddle cells and wall
cells; two and three tiles in flight; coarse levels of ratio 2, 3 and 1; one
cell across an axis; every wall type as the end of a path; a field that is
rough from cell to cell, so that a ray that enters a wrong cell shows."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W

pytestmark = pytest.mark.gpu

TAB = dict(nB=21, nQ=5, nT=17)

CASES = {
    # 2 chunks of one (cell, replicate): 16 of them in a tile, carries in every axis
    "carry": dict(n=(5, 3, 7), photmax=7, nVar=3),
    "carry_one_wide": dict(n=(1, 1, 9), photmax=1, nVar=1),
    "carry_one_row": dict(n=(33, 1, 2), photmax=3, nVar=2),
    # 32 chunks (5 of them padding), then 64 (one tile and a half)
    "one_cell_tiles": dict(n=(6, 5, 4), photmax=107, nVar=2),
    "two_tiles_a_cell": dict(n=(4, 3, 2), photmax=150, nVar=2),
    "walls_straddle": dict(n=(7, 5, 3), photmax=9, nVar=3, calcwalls=1, adiabw=1, adiabe=1),
    "ratio3": dict(n=(9, 6, 12), photmax=33, nVar=2, levels=[(9, 6, 12), (3, 2, 4)], maxs=[2, 100000], calcwalls=1,
                   adiabw=1),
    "ratio_mixed": dict(n=(8, 6, 4), photmax=20, nVar=2, levels=[(8, 6, 4), (4, 2, 4), (2, 1, 2)], maxs=[1, 3, 100000],
                        bd_y=3, bd_z=2),
    "no_fine_steps": dict(n=(8, 8, 8), photmax=16, nVar=2, levels=[(8, 8, 8), (4, 4, 4)], maxs=[0, 40]),
    "black_yz": dict(n=(8, 6, 5), photmax=25, nVar=2, bd_y=2, bd_z=2, calcwalls=1, adiabe=1),
    "specular_yz": dict(n=(6, 7, 8), photmax=25, nVar=2, bd_y=3, bd_z=3),
    "grey_long": dict(n=(13, 11, 9), photmax=40, nVar=2, grey=True),
}


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_tiles_and_cells_equal_the_oracle(name, fp64):
    from oracle import oracle as O
    c = dict(CASES[name])
    im, jm, km = c.pop("n")
    p = W.channel_params(im, jm, km, floatpoint=fp64, **dict(TAB, **c))
    tabs = None if p.grey else W.tables_nb(**TAB)
    rng = np.random.default_rng(len(name))
    T = (W.channel_field(p, seed=5) + rng.uniform(-25, 25, api.field_shape(p))).astype(np.float32)
    s = api.Solver(p, tabs)
    for rpt in (2, 4, 8):     # three tiles in flight up to 4, two above
        s.set_launch(rays_per_thread=rpt)
        t = s.solve_async(T)
        steps = s.info(t).steps
        r = s.collect(t)
        o = O.solve(p, tabs, T, rpt=rpt, fp64=bool(fp64))
        for k in ("q64", "var64", "qw64", "vw64"):
            np.testing.assert_array_equal(getattr(r, k), o[k], err_msg="%s rpt %d" % (k, rpt))
        assert steps == o["steps"]
    s.close()


def test_scattering_tiles_equal_the_oracle():
    from oracle import oracle as O
    p = W.channel_params(9, 6, 12, photmax=19, nVar=3, levels=[(9, 6, 12), (3, 2, 4)], maxs=[3, 100000], bd_y=3,
                         calcwalls=1, adiabw=1, adiabe=1, **TAB)
    tabs = W.tables_nb(**TAB)
    rng = np.random.default_rng(3)
    T = (W.channel_field(p, seed=5) + rng.uniform(-25, 25, api.field_shape(p))).astype(np.float32)
    s = api.Solver(p, tabs)
    sc = api.Scattering.synthetic(nB=TAB["nB"], nQ=TAB["nQ"], nA=31, ksca_lo=0.5, ksca_hi=8.0, g_lo=-0.4, g_hi=0.8)
    s.set_scattering(sc)
    r = s.solve(T)
    o = O.solve(p, tabs, T, rpt=s.get_launch()[0], scatter=sc.arrays())
    np.testing.assert_array_equal(r.q64, o["q64"])
    np.testing.assert_array_equal(r.qw64, o["qw64"])
    s.close()
