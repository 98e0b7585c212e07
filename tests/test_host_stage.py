"""The page-locked staging buffers and copy threads that every handle of a process shares (csrc/host_stage.h), without a
GPU: a small program against the header, with fakes for the CUDA calls it makes."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="session")
def program(tmp_path_factory):
  out = str(tmp_path_factory.mktemp("native") / "host_stage_test")
  cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
  subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-Wall", "-pthread", "-I", os.path.join(cuda, "include"),
                         "-I", os.path.join(ROOT, "cuhnsw_b200", "csrc"),
                         os.path.join(ROOT, "tests", "native", "host_stage_test.cpp"), "-o", out, "-ldl"])
  return out


@pytest.mark.parametrize("check", ["users", "thread-limit", "fork", "unwinding"])
def test_host_stage(program, check):
  subprocess.run([program, check], check=True, timeout=60)
