"""Launchers of the lattice passes on a stand-in CUDA runtime (no device): every pass launches
on the first device that a process uses and on the next one, whose kernels start with their
own limits of shared memory; and whatever table the last ensemble was made with."""
from __future__ import annotations

import pathlib
import shutil
import subprocess

import pytest

import misa_b200 as mb

ROOT = pathlib.Path(__file__).resolve().parents[1]
PKG = ROOT / "misa-md-hip_b200"
OBJECTS = ("mb_kernels64", "mb_split64", "mb_shell64", "mb_geometry", "mb_ensemble_split", "mb_ensemble")


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    out = tmp_path_factory.mktemp("launches") / "driver"
    mb.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = ROOT / "tests" / "launches"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--cudart", "none",
                    f"-I{PKG / 'csrc'}", f"-I{ROOT / 'include'}", str(src / "driver.cu"), str(src / "runtime.cpp"),
                    *[str(PKG / "_build" / f"{o}.o") for o in OBJECTS], "-o", str(out)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    return [line.split() for line in r.stdout.split("\n") if line]


@pytest.mark.parametrize("device", ["0", "1"])
def test_every_pass_launches_on_every_device(lines, device):
    got = [(name, status) for d, name, status in lines if d == device]
    assert len(got) == 44
    assert all(status == "0" for _, status in got), [g for g in got if g[1] != "0"]
