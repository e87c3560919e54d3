"""The page-locked ring's transfers, failed ones included, without a GPU: tests/c_abi/host_stage.cpp on a CUDA runtime of its own."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.join(ROOT, "tests", "c_abi")


def test_source_is_not_read_after_the_call(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = os.path.join(str(tmp_path), "host_stage")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-pthread", "-I", os.path.join(HERE, "fake_cuda"), "-I", os.path.join(ROOT, "z-ant_b200", "csrc"),
                           os.path.join(HERE, "host_stage.cpp"), "-o", exe])
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout)


def test_no_stream_is_used_after_it_was_left(tmp_path):
    """A context's change of stream (leave_stream, what zant_b200_ctx_set_stream does) between transfers of every kind."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = os.path.join(str(tmp_path), "host_stage")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-pthread", "-I", os.path.join(HERE, "fake_cuda"), "-I", os.path.join(ROOT, "z-ant_b200", "csrc"),
                           os.path.join(HERE, "host_stage.cpp"), "-o", exe])
    r = subprocess.run([exe, "streams"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout)
