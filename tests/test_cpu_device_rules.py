"""Integer rules of the device code that decide whether an access stays in
bounds, compiled for the host and run over their ranges (tests/c/device_rules.cu):
a cell's table coordinate against the codes of the halo, and an emitted
bundle's packed cell and the offset of a cell in a large pyramid, whose limits
the parameter check keeps."""
import os
import subprocess

import pytest

from radchan_b200 import api
from radchan_b200 import build as B
from radchan_b200 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rules") / "device_rules")
    cmd = [B.NVCC] + B.ARCH + ["-std=c++17", "-O1", "-I" + B.INCLUDE, "-I" + B.CSRC,
                               os.path.join(HERE, "c", "device_rules.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    return r.stdout


@pytest.mark.parametrize("name", ["coords", "offsets", "packing"])
def test_rule_holds(rules, name):
    assert "ok " + name in rules.splitlines(), rules


@pytest.mark.parametrize("axis", ["imax", "jmax", "kmax"])
def test_edges_beyond_the_packed_cell_are_refused(axis):
    at = ["imax", "jmax", "kmax"].index(axis)
    for edge, ok in ((32767, True), (32768, True), (65535, True), (65536, False), (131072, False)):
        n = [4, 4, 4]
        n[at] = edge
        msg = api.validate(W.channel_params(*n, grey=True))
        assert (msg == "") == ok, (edge, msg)
        assert ok or axis in msg


def test_table_dimensions_beyond_the_packed_band_are_refused():
    for kw, ok in ((dict(nB=1 << 20, nQ=1, nT=2), True), (dict(nB=(1 << 20) + 1, nQ=1, nT=2), False),
                   (dict(nB=2, nQ=2048, nT=2), True), (dict(nB=2, nQ=2049, nT=2), False),
                   (dict(nB=32767, nQ=256, nT=256), True), (dict(nB=32768, nQ=256, nT=256), False)):
        assert (api.validate(W.channel_params(8, 8, 8, **kw)) == "") == ok, kw
    p = W.channel_params(8, 8, 8, grey=True)
    p.grey_nB = (1 << 20) + 1
    assert "bands" in api.validate(p)


def test_the_largest_grids_are_those_whose_pyramid_has_32_bit_offsets():
    for n, ok in (((1289, 1289, 1289), True), ((1290, 1290, 1290), True), ((1291, 1291, 1291), False),
                  ((30000, 35000, 2), True), ((30000, 36000, 2), False), ((65535, 32767, 1), False),
                  ((1, 1, 65535), True)):
        msg = api.validate(W.channel_params(*n, grey=True))
        assert (msg == "") == ok, (n, msg)
    lv = [(1200, 1200, 1200), (600, 600, 600), (300, 300, 300)]
    assert api.validate(W.channel_params(*lv[0], grey=True, levels=lv, maxs=[5, 5, 100])) == ""
    lv = [(1280, 1280, 1280), (640, 640, 640), (320, 320, 320)]
    assert "32-bit" in api.validate(W.channel_params(*lv[0], grey=True, levels=lv, maxs=[5, 5, 100]))
