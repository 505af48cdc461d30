"""The status of a failed resident search (csrc/search_error.h): an expired wait is a timeout, as it is
for the counters, everything else a broken invariant.  (No wait is made to run out on a GPU.)"""
import os
import shutil
import subprocess

import pytest

import tensorfim_b200 as tf

CSRC = os.path.join(os.path.dirname(os.path.abspath(tf.__file__)), "csrc")


def test_status_of_a_failed_search(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    src, exe = tmp_path / "e.cpp", tmp_path / "e"
    src.write_text('#include "search_error.h"\nint main() { using namespace tfim;\n'
                   "return search_error_status(0) == TFIM_OK && search_error_status(kErrRow) == TFIM_E_STATE &&\n"
                   "search_error_status(kErrProjected) == TFIM_E_STATE && search_error_status(kErrWait) == TFIM_E_TIMEOUT ? 0 : 1; }\n")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", os.path.join(CSRC, "..", "..", "include"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0
    with open(os.path.join(CSRC, "resident.cu")) as f:
        s = f.read()
    # both wave loops report through it, and the barrier's expiry is recorded as such
    assert s.count("check_search(c, hst->error)") == 2 and s.count("atomicExch(&st->error, kErrWait)") == 3
    assert "search_error_status(error)" in s
