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
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-rdynamic", f"-I{os.path.join(REPO, 'nyx_gb300', 'csrc')}",
                    os.path.join(REPO, "tests", "c_abi", "pages_driver.cpp"), "-o", str(exe), "-lpthread"], check=True)

    def run(what):
        r = subprocess.run([str(exe), what], capture_output=True, text=True, timeout=120)
        return r.returncode, r.stdout
    return run


@pytest.mark.parametrize("what", ["keeps", "refused"])
def test_pages_come_in_and_nothing_is_written(driver, what):
    assert driver(what) == (0, "ok\n")
