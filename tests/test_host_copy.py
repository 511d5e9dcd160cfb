"""The host side of the transfers (csrc/host_copy.h), compiled with a stand-in for the CUDA runtime that reads
and writes pinned memory as late as the real one may."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path_factory.mktemp("host_copy") / "host_copy_check")
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-g", "-pthread", "-Wno-unused-function", "-o", exe,
                           os.path.join(ROOT, "tests", "host_copy_check.cpp"), "-ldl"])

    def run(*what, **env):
        r = subprocess.run([exe, *what], env=dict(os.environ, **env), capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_upload_sources_are_the_callers_again(check):
    check("upload_sources")


def test_downloads_and_the_ring_behind_a_failed_one(check):
    check("downloads")


@pytest.mark.parametrize("asked,granted,expected", [("3", 9, 3), ("1", 9, 1), ("0", 9, 0), ("7", 9, 3), ("-1", 9, 0),
                                                    ("3", 0, 0), ("3", 1, 1)])
def test_helper_threads_asked_for_and_granted(check, asked, granted, expected):
    """Threads the system refuses are done without: no exception, no lock left behind."""
    check("helpers", str(granted), str(expected), COLI_CUDA_COPY_THREADS=asked)


def test_helper_threads_by_default(check):
    check("helpers", "9", str(min(3, len(os.sched_getaffinity(0)) // 4)), COLI_CUDA_COPY_THREADS="")


@pytest.mark.parametrize("asked", ["3", "0"])
def test_several_threads_copy_at_once(check, asked):
    check("many_callers", COLI_CUDA_COPY_THREADS=asked)


def test_transfers_without_pinned_memory(check):
    check("no_pinned_memory")


def test_rows_of_a_blocking_call_in_pieces(check):
    check("row_pieces")


def test_ring_of_several_threads(check):
    check("ring_of_several_threads")
