"""The shared host copies on a stand-in CUDA runtime (no device): when a call or an allocation
under them fails every copy still succeeds with the right bytes, and all that was taken is
given back; copies of every size from 2 MiB on go through the slots once they are there."""
from __future__ import annotations

import os
import pathlib
import shutil
import subprocess

import pytest

import misa_b200 as mb

ROOT = pathlib.Path(__file__).resolve().parents[1]
PKG = ROOT / "misa-md-hip_b200"


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_copy") / "driver"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = pathlib.Path(nvcc).resolve().parents[1] / "include"
    mb.build()
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{PKG / 'csrc'}", f"-I{ROOT / 'include'}", f"-I{include}",
                    str(ROOT / "tests" / "host_copy" / "driver.cpp"), str(PKG / "_build" / "mb_host_copy.o"),
                    "-lpthread", "-ldl", "-o", str(out)], check=True, capture_output=True, text=True)
    return out


@pytest.mark.parametrize("scenario", ["none", "event", "memory 0", "memory 1", "memory 2", "memory 4"])
def test_copies_survive_a_failing_call(driver, scenario):
    r = subprocess.run([str(driver), *scenario.split()], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.split("\n")
    assert lines[:3] == ["0 1 0 1"] * 3, lines
    assert lines[3] == "left 0 0"


@pytest.mark.skipif((os.cpu_count() or 1) < 4, reason="one thread copies plainly")
def test_copies_of_every_size_take_the_slots_that_are_there(driver):
    sizes = [2, 3, 7, 8, 14, 31]  # MiB and a short last chunk: fewer chunks than slots, as many, more
    r = subprocess.run([str(driver), "sizes", *map(str, sizes)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.split("\n")
    for k, mib in enumerate(sizes):
        assert lines[3 + 2 * k] == "0 1 0 1", mib
        assert lines[4 + 2 * k] == f"pieces {2 * (mib + 1)}", mib  # up and down
