"""A plan run that fails half-way leaves the caller's stream behind every
launch already queued on the plan's side streams (csrc/stream_fork.h), shown
with a runtime that keeps account of the orderings: a later launch fails, or
any one of the ordering calls does."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = tmp_path_factory.mktemp("fork") / "fork_host"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(cuda, "include"),
                           "-I", os.path.join(ROOT, "molscat_b200", "csrc"),
                           os.path.join(ROOT, "tests", "host", "fork_host.cpp"), "-o", str(exe)])
    return str(exe)


def test_a_run_without_errors_is_joined(host):
    subprocess.check_call([host])


def test_a_failed_launch_is_joined(host):
    subprocess.check_call([host, "0", "launch"])


@pytest.mark.parametrize("call", range(1, 10))
@pytest.mark.parametrize("launch", [[], ["launch"]])
def test_a_failed_ordering_call_is_joined(host, call, launch):
    subprocess.check_call([host, str(call), *launch])


def test_the_run_uses_it():
    with open(os.path.join(ROOT, "molscat_b200", "csrc", "propagator.cu")) as f:
        src = f.read()
    body = src[src.index("int mgpu_plan_run_device_phases(mgpu_plan *p"):]
    body = body[:body.index("\n}\n")]
    assert "StreamFork fork(st, p->ev_in)" in body
    assert "cudaStreamWaitEvent" not in body and "cudaEventRecord" not in body
