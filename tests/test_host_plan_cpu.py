"""The host plan's own logic (opencnn_b200/csrc/host_plan.h) without a GPU: tests/host_plan_fake.cpp compiles it against a runtime whose
streams run in any order that their events allow and whose calls can be made to fail."""
import os
import subprocess

import pytest

from opencnn_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="session")
def host_plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_plan") / "host_plan_fake")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", include, "-o", exe, os.path.join(HERE, "host_plan_fake.cpp")], check=True)
    return lambda *args: subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120).stdout.strip()


@pytest.mark.parametrize("check", ["results", "errors", "apart", "streams", "no_streams", "overlap"])
def test_host_plan(host_plan, check):
    assert host_plan(check) == "ok"


def test_the_banded_plans_of_the_gpu_tests_are(host_plan):
    from test_parity_gpu import BANDED
    for _, (N, C, K, H, W) in BANDED:
        assert int(host_plan("bands", N, C, H, W, K)) > 1, (N, C, K, H, W)
    assert int(host_plan("bands", 32, 16, 12, 12, 64)) == 1
