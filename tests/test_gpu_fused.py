"""Deferred elementwise ops (one kernel per chain) against the oracle, which computes op by op: chains whose program is compiled
ahead of time and ones that are interpreted, groups of four elements and single ones, windows, broadcasts and reductions in
between, operands changed in place between an op and its evaluation."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import assert_close

pytestmark = pytest.mark.gpu

# one element; rows of fewer / exactly / more than four; an odd row length; one tile of 512 elements and one more; above the size
# up to which shared intermediate results are kept
SHAPES = [(1, 1), (3, 3), (5, 4), (7, 36), (64, 577), (4, 128), (3, 171), (1100, 1000)]


@pytest.fixture(scope="module")
def engines():
    import rusttensor_b200

    return rusttensor_b200.engine(), oracle.engine()


def chain(e, x, b, col):
    o = e.ops
    rows, cols = x.shape
    t = o.tanh(o.add(o.mul(x, b), col))
    u = o.div(o.sin(x), o.add(o.square(x), e.tensor(np.float32(1.5), ())))
    v = o.elu(o.clip(o.sub(t, u), -0.7, 0.9), 0.5)
    w = o.slice(o.softplus(v), [(0, rows), (cols // 2, cols)])
    z = o.concat([w, o.sigmoid(x), w], 1)
    return o.maximum(o.mul_scalar(z, -0.5), o.exp(o.mul_scalar(o.square(z), -1.0))), t, v


@pytest.mark.parametrize("shape", SHAPES)
def test_chain_forward_and_backward(engines, shape):
    r = np.random.default_rng(shape[0] * 31 + shape[1])
    data = [r.standard_normal(s).astype(np.float32) for s in (shape, shape[1:], (shape[0], 1))]
    out = []
    for e in engines:
        x, b, col = (e.tensor(d, requires_grad=True) for d in data)
        y, t, v = chain(e, x, b, col)
        loss = e.ops.add(e.ops.mean(y), e.ops.sum(e.ops.logsumexp(v, 1)))
        loss.backward()
        out.append([y, v, t, loss] + [p.grad for p in (x, b, col)])
    for got, ref in zip(*out):
        assert_close(got.numpy(), ref.numpy())


@pytest.mark.parametrize("shape", SHAPES[:-1])
def test_operands_changed_in_place_after_the_op(engines, shape):
    r = np.random.default_rng(7)
    a, b = (r.standard_normal(shape).astype(np.float32) for _ in range(2))
    out = []
    for e in engines:
        x = e.tensor(a, requires_grad=True)
        y = e.ops.exp(e.ops.mul_scalar(x, 0.5))  # not asked for before x changes
        loss = e.ops.mean(e.ops.square(x))
        loss.backward()
        x.update_from_host(b)
        z = e.ops.tanh(x)
        e.Sgd([x], 0.1).step()
        out.append([y, z, x])
    for got, ref in zip(*out):
        assert_close(got.numpy(), ref.numpy())


@pytest.mark.parametrize("written", ["base", "slice", "slice of a slice"])
def test_rows_and_their_base_written_through_a_device_pointer(capi, written):
    import rusttensor_b200

    e, data = rusttensor_b200.engine(), np.arange(24, dtype=np.float32).reshape(6, 4)
    x = e.tensor(data)
    y = e.ops.slice(x, [(1, 5), (0, 4)])
    y.numpy()
    w = e.ops.slice(y, [(2, 3), (0, 4)])
    w.numpy()
    z = e.ops.square(y)  # not asked for before the write
    tensors = {"base": x, "slice": y, "slice of a slice": w}
    p, other = C.c_void_p(), np.full(tensors[written].shape, -77, np.float32)
    e._call("tensor_device_ptr", C.c_int64(tensors[written].handle), C.byref(p))
    capi.call("memcpy_h2d", p, other.ctypes.data_as(C.c_void_p), C.c_size_t(other.nbytes))
    for name, want in (("base", data), ("slice", data[1:5]), ("slice of a slice", data[3:4])):
        np.testing.assert_array_equal(tensors[name].numpy(), other if name == written else want)
    np.testing.assert_array_equal(z.numpy(), data[1:5] ** 2)


@pytest.mark.parametrize("rows,classes", [(1, 2), (7, 16), (33, 17), (64, 65), (5, 300)])
@pytest.mark.parametrize("steps", [1, 2, 205])
def test_losses_of_a_sequence(engines, rows, classes, steps):
    r = np.random.default_rng(rows + classes + steps)
    h = r.standard_normal((steps, rows, 9)).astype(np.float32)
    w, bias = r.standard_normal((9, classes)).astype(np.float32), r.standard_normal(classes).astype(np.float32)
    y = np.eye(classes, dtype=np.float32)[r.integers(0, classes, (steps, rows))]
    out = []
    for e in engines:
        tw, tb = e.tensor(w, requires_grad=True), e.tensor(bias, requires_grad=True)
        total = None
        for t in range(steps):
            logits = e.ops.add(e.ops.matmul(e.tensor(h[t]), tw), e.ops.broadcast_to(tb, (rows, classes)))
            loss = e.ops.softmax_cross_entropy(logits, e.tensor(y[t]), 1)
            total = loss if total is None else e.ops.add(total, loss)
        total.backward()
        out.append([total, tw.grad, tb.grad])
    for got, ref in zip(*out):
        assert_close(got.numpy(), ref.numpy())


def test_a_malformed_program_is_refused():
    from rusttensor_b200 import CApi
    from rusttensor_b200.capi import RtError

    api = CApi()
    with pytest.raises(RtError):
        api.call("fused_elementwise", C.create_string_buffer(8192))  # zero dimensions, no outputs
    api.close()


# one block and several, a row more and less than a block of each form (128 rows; 8 rows), the change of form at 16 classes
@pytest.mark.parametrize("rows,classes", [(1, 1), (127, 10), (129, 16), (9, 17), (1000, 16), (64, 65), (9, 128), (1003, 129), (300, 300)])
def test_classification_loss_with_gradient(rows, classes):
    import ctypes as C

    from rusttensor_b200 import CApi

    api, r = CApi(), np.random.default_rng(rows + classes)
    x, t = r.standard_normal((rows, classes)).astype(np.float32), r.random((rows, classes), dtype=np.float32)
    dx, dt, loss, grad = api.to_device(x), api.to_device(t), api.to_device(np.zeros(1, np.float32)), api.to_device(np.zeros_like(x))
    ls = x - np.log(np.exp(x.astype(np.float64)).sum(1, keepdims=True))
    for _ in range(2):  # the ticket has to be back at zero
        api.call("softmax_nll_with_grad", dx.ptr, dt.ptr, C.c_int64(rows), C.c_int64(classes), C.c_float(-1), C.c_float(rows), None, C.c_float(-1 / rows),
                 loss.ptr, grad.ptr)
        np.testing.assert_allclose(loss.numpy()[0], -(ls * t).sum() / rows, rtol=2e-6, atol=1e-7)
        want = -(t - np.exp(ls) * t.sum(1, keepdims=True, dtype=np.float64)) / rows
        np.testing.assert_allclose(grad.numpy(), want, rtol=1e-4, atol=2e-6 * np.abs(want).max() + 1e-9)
    api.close()


def program_counts(capi):
    n = C.c_int64(0), C.c_int64(0)
    capi.call("fused_launch_counts", C.byref(n[0]), C.byref(n[1]))
    return n[0].value, n[1].value, capi.launches()


# A changed order of a program's instructions or registers would miss every compiled program without a wrong value: the steps of the
# workloads have to find theirs.  The recurrent ones have none in a capture (one from the fused ops is interpreted); what has to hold there is that
# the step is a handful of launches, however many timesteps it has.
@pytest.mark.parametrize("config,dims,interpreted,launches", [(1, [64, 784, 128, 10], 0, 9), (101, [7, 13, 5, 3], 0, 10), (2, [33, 57], 0, 4),
                                                              (2, [1100, 1000], 0, 4), (3, [16, 28, 32, 64, 128, 10], 0, 21),
                                                              (103, [5, 8, 3, 4, 7, 3], 0, 23), (4, [2, 3, 6, 5], 0, 22), (104, [8, 64, 56, 128], 0, 27),
                                                              (5, [50, 200, 60, 30], 0, 15), (105, [50, 200, 60, 30], 1, 14), (5, [50, 200, 120, 30], 0, 15),
                                                              (105, [50, 200, 120, 30], 1, 16)])
def test_the_workloads_find_their_compiled_programs(capi, config, dims, interpreted, launches):
    import rusttensor_b200

    tr = rusttensor_b200.DataParallelTrainer(config, dims)
    rusttensor_b200.engine()._call("sync")  # what others have left unevaluated is none of the step's
    before = program_counts(capi)
    tr.capture()
    found, missed, launched = (b - a for a, b in zip(before, program_counts(capi)))
    assert missed <= interpreted and (found >= 1 or config % 100 == 5) and launched <= launches, (found, missed, launched)


def test_timesteps_that_are_not_captured_find_theirs(capi):
    import rusttensor_b200
    from helpers import workload_data

    dims = [50, 200, 60, 30]
    tr = rusttensor_b200.DataParallelTrainer(5, dims)
    before = program_counts(capi)
    tr.step_eager(workload_data(5, dims, seed=0)[1])
    found, missed, _ = (b - a for a, b in zip(before, program_counts(capi)))
    assert missed <= 6 and found >= 4 * dims[2], (found, missed)  # the first and last timesteps are interpreted
