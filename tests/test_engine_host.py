"""Host logic of the CUDA backend that needs no GPU: tests/host/engine_checks.cpp over stubs of the C ABI."""
import os
import re
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


@pytest.mark.parametrize("name", ["cells_become_a_sequence", "long_recurrences", "recurrences_have_their_values", "gradients_of_rows", "logsumexps_are_computed", "refused_programs_take_no_memory", "a_capture_in_two_parts", "kept_results_stay_where_they_are_written", "rows_do_not_alias", "rows_in_a_capture", "broadcast_does_not_alias", "pooling_knows_its_relu", "errors_lose_nothing", "written_from_outside", "a_product_of_a_matrix_with_itself"])
def test_engine(checks, name):
    r = subprocess.run([checks, name], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, f"exit code {r.returncode}\n{r.stdout}{r.stderr}"


def test_kernel_attributes_are_set_on_every_device(tmp_path):
    """An attribute of a kernel belongs to a device: the helper that sets it sets it on each, and no source file keeps the answer in a
    static of its own."""
    exe, csrc = tmp_path / "device_once", os.path.join(os.path.dirname(HERE), "rusttensor_b200", "csrc")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", str(exe),
                    os.path.join(HERE, "host", "device_once_checks.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    for name in os.listdir(csrc):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(csrc, name)) as f:
                assert not re.search(r"static\s+(const\s+)?(cudaError_t|auto|int|bool)\s+\w+\s*=[^;]*cuda(FuncSetAttribute|Occupancy)", f.read()), name


def test_both_gradients_of_parts_launch_all_or_nothing(tmp_path):
    obj, exe = str(tmp_path / "parts.o"), str(tmp_path / "parts_checks")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "-c",
                    os.path.join(os.path.dirname(HERE), "rusttensor_b200", "csrc", "k_gemm_parts.cu"), "-o", obj], check=True)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", exe,
                    os.path.join(HERE, "host", "parts_checks.cpp"), obj], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_piece_of_mail_is_one_element_of_its_access():
    """A vector access is one access per element, in no order.  Where blocks tell one another values beside a number that says which timestep they
    are of (the backward recurrence), both are halves of one 64-bit element; forward the number is a bit of the 32-bit value."""
    with open(os.path.join(os.path.dirname(HERE), "rusttensor_b200", "csrc", "k_lstm_seq.cu")) as f:
        source = f.read()
    forward, backward = source.split("lstm_sequence_backward_kernel(const SeqArgs a) {", 1)
    accesses = [(re.findall(r"__forceinline__ \S+ (\w+)\(", source[: m.start()])[-1], m.group()) for m in re.finditer(r"(ld|st)\.relaxed\.[\w.]+", source)]
    assert sorted(accesses) == [("peek", "ld.relaxed.gpu.global.v4.u32"), ("peek2", "ld.relaxed.gpu.global.v2.b64"),
                                ("post2", "st.relaxed.gpu.global.v2.b64"), ("post_output", "st.relaxed.gpu.global.u32")]
    forward = forward[forward.index("lstm_sequence_kernel(const SeqArgs a) {"):]
    assert re.findall(r"a, (peek2?), \[", forward) == ["peek"] and "post2" not in forward
    assert re.findall(r"a, (peek2?), \[", backward) == ["peek2"] and "post_output" not in backward
