"""Host logic of the CUDA backend that needs no GPU: tests/host/engine_checks.cpp over stubs of the C ABI."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    exe = tmp_path_factory.mktemp("engine_checks") / "engine_checks"
    # entry points that no check reaches stay undefined
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-no-pie", "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe),
                    os.path.join(HERE, "host", "engine_checks.cpp")], check=True)
    return str(exe)


@pytest.mark.parametrize("name", ["rows_do_not_alias", "rows_in_a_capture", "pooling_knows_its_relu", "errors_lose_nothing"])
def test_engine(checks, name):
    r = subprocess.run([checks, name], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, f"exit code {r.returncode}\n{r.stdout}{r.stderr}"
