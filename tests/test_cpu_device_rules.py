"""Integer rules of the device code that decide whether an access stays in
bounds, compiled for the host and run over their ranges (tests/c/device_rules.cu):
a cell's table coordinate against the codes of the halo."""
import os
import subprocess

import pytest

from radchan_b200 import build as B

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


@pytest.mark.parametrize("name", ["coords"])
def test_rule_holds(rules, name):
    assert "ok " + name in rules.splitlines(), rules
