"""CPU: the host-buffer calls' slicing, ordering and fallbacks, in a program that
builds their source with the host compiler against a stand-in CUDA runtime
(tests/cpp/host_path_test.cpp) and the oracle's codec."""
import os
import subprocess

import pytest

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    oracle.build(with_reference=False)
    exe = str(tmp_path_factory.mktemp("host") / "host_path_test")
    lib = os.path.join(ROOT, "oracle")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-pthread", "-I", os.path.join(CUDA, "include"),
                    "-x", "c++", os.path.join(ROOT, "frsz_b200", "csrc", "frsz2_host.cu"),
                    os.path.join(ROOT, "tests", "cpp", "host_path_test.cpp"), "-x", "none",
                    os.path.join(lib, "libfrsz2_oracle.so"), f"-Wl,-rpath,{lib}", "-o", exe, "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["plain", "pending_pinned", "pending_pageable", "no_slots", "some_slots",
                                      "throwing"])
def test_scenario(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
