"""The host pages of a buffer that a read-back will fill (nyx_gb300/csrc/pm_pages.h), in a
small C++ program: no GPU."""
from __future__ import annotations

import os
import subprocess

import pytest

from tests.conftest import REPO


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pages") / "pages_driver"
    src = os.path.join(REPO, "tests", "c_abi", "pages_driver.cpp")
    include = os.path.join(REPO, "nyx_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-rdynamic", f"-I{include}", src, "-o", str(exe),
                    "-lpthread", "-ldl"], check=True)

    def run(what):
        r = subprocess.run([str(exe), what], capture_output=True, text=True, timeout=120)
        return r.returncode, r.stdout
    return run


@pytest.mark.parametrize("what", ["keeps", "there", "refused"])
def test_pages_come_in_and_nothing_is_written(driver, what):
    assert driver(what) == (0, "ok\n")


@pytest.mark.parametrize("what", ["memory", "threads"])
def test_threads_that_cannot_be_had(driver, what):
    assert driver(what) == (0, "ok\n")
