"""CPU test of the threads that fill the pinned buffer of a dispatch
(csrc/host_copy.h), compiled with g++."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ is missing")
    out = str(tmp_path_factory.mktemp("hc") / "host_copy_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", out, os.path.join(HERE, "host_copy_host.cpp")],
                   check=True)
    return out


def _run(exe, *args):
    r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=60)
    return r.returncode, r.stdout.strip()


@pytest.mark.parametrize("extra", [0, 1, 3, 7])
@pytest.mark.parametrize("megabytes", [0, 1, 9, 40])
def test_every_byte_arrives_in_order(exe, extra, megabytes):
    assert _run(exe, extra, -1, megabytes) == (0, "ok")


def test_memory_that_runs_out_while_threads_are_made(exe):
    """From the first allocation that fails on, the call either reports it
    before any thread runs or copies everything with the threads it has."""
    out = [_run(exe, 7, k, 9) for k in range(60)]
    assert all(rc == 0 for rc, _ in out), out
    assert out[0][1] == "no memory" and out[-1][1] == "ok"
