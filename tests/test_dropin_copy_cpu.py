"""The drop-in entries' copies (csrc/dropin_copy.cu) over a stand-in for the
CUDA runtime (dropin_copy_check.cpp): what a call leaves behind when a runtime
call fails, and which arrays the threads may take."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "nr-amssncku_b200")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")) or not shutil.which("g++"):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("copy") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", include, "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(os.path.dirname(PKG), "include"), "-x", "c++",
                    os.path.join(HERE, "dropin_copy_check.cpp"), os.path.join(PKG, "csrc", "dropin_copy.cu"),
                    "-o", exe, "-lpthread"], check=True)
    return exe


# works: the threaded form itself.  copy_fails, wait_fails: one worker's copy
# or wait fails while the others have pieces in flight.  The others: arrays that
# are not ordinary host memory, all of them or some, a null pointer, and output
# arrays that share memory or just do not; a caller that changes its device; and
# calls from many threads, one after another and at once
@pytest.mark.parametrize("scenario", ["works", "copy_fails", "wait_fails", "pinned", "managed", "some_pinned",
                                      "few_pageable", "device", "null", "same_array", "overlap", "adjacent",
                                      "devices", "thread_a_call", "threads_at_once"])
def test_copies(check, scenario):
    r = subprocess.run([check, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)
