"""Failing calls of the CUDA runtime and of the thread library, injected by a fake of both (tests/kat/runtime_kat.cpp), in
the host runtime: nothing here touches a GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gpu-path-tracer_b200", "csrc")


@pytest.fixture(scope="module")
def runtime_kat(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("kat") / "runtime_kat")
    subprocess.run(["g++", "-O1", "-std=c++17", "-rdynamic", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "kat", "runtime_kat.cpp"), "-o", out, "-ldl", "-lpthread"], check=True)
    return out


@pytest.mark.parametrize("case", [
    "upload", "upload without pinned memory", "upload without streams", "upload without the last stream",
    "upload without events", "upload without threads", "upload with two threads", "upload that fails", "two uploads at once",
    "a batch whose second launch fails", "a batch that cannot be waited for", "batches of many threads"])
def test_runtime_with_failing_calls(runtime_kat, case):
    p = subprocess.run([runtime_kat, case], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr
