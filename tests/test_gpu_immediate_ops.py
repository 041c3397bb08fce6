"""The engine with deferral off: every op by its own kernel at once, which otherwise only tensors of 2^31 and more elements reach.  The
parity tests of the ops and of the workloads, run that way."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_ops_parity import *  # noqa: F401,F403
from test_gpu_workloads import test_fused_forward_ops_match_the_reference_chain, test_small_workload_matches_oracle  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def immediate_ops(gpu_engine):
    gpu_engine._call("set_deferred_ops", C.c_int(0))
    yield
    gpu_engine._call("set_deferred_ops", C.c_int(1))


def launches(capi):
    n = C.c_int64(0)
    capi.call("kernel_launch_count", C.byref(n))
    return n.value


def test_an_op_is_one_launch_at_once(gpu_engine, capi):
    x = gpu_engine.tensor(np.ones((5, 3)), requires_grad=True)
    before = launches(capi)
    y = gpu_engine.ops.square(gpu_engine.ops.exp(x))
    assert launches(capi) == before + 2
    gpu_engine._call("set_deferred_ops", C.c_int(1))
    z = gpu_engine.ops.square(gpu_engine.ops.exp(x))
    assert launches(capi) == before + 2
    gpu_engine._call("set_deferred_ops", C.c_int(0))  # what was deferred is done first
    assert launches(capi) > before + 2
    np.testing.assert_array_equal(y.numpy(), z.numpy())
