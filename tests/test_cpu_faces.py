"""The march computes a y or z face as float(index) * spacing instead of
loading it: the grid the library builds holds exactly that product."""
import numpy as np
import pytest

from radchan_b200 import api
from radchan_b200 import workloads as W


@pytest.mark.parametrize("edges", [(8, 6, 4), (45, 27, 33), (64, 64, 64), (17, 193, 127)])
def test_yz_faces_are_index_times_spacing(edges):
    p = W.channel_params(*edges, grey=True)
    g = api.grid_level(p, 0)
    for name, L, n in (("yu", p.Ly, edges[1]), ("zu", p.Lz, edges[2])):
        d = np.float32(np.float32(L) / np.float32(n))
        np.testing.assert_array_equal(g[name], np.arange(n + 1).astype(np.float32) * d)
