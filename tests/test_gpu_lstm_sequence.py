"""The recurrence of a whole sequence in one kernel (rt_lstm_sequence and its gradient) against float64: batches and hidden sizes at the
edges of the blocks' 16 rows and 8 / 16 units, given and zero initial states, a strided weight matrix, and sizes that run timestep by
timestep because their blocks would not all be resident."""
import ctypes as C

import numpy as np
import pytest

import rusttensor_b200
from helpers import assert_close, rng, workload_data

pytestmark = pytest.mark.gpu

i64 = C.c_int64
# (steps, batch, hidden); the last two do not fit
SIZES = [(1, 1, 1), (2, 16, 8), (5, 17, 9), (3, 15, 64), (7, 30, 200), (4, 33, 129), (9, 64, 512), (3, 8, 1000), (3, 90, 512), (2, 40, 700)]


def sigmoid(v):
    return 1 / (1 + np.exp(-v))


def reference(pre, w, h, c, dh_all, steps, batch, hidden):
    pre, w, h, c, dh_all = (v.astype(np.float64) for v in (pre, w, h, c, dh_all))
    hs, kept = [], []
    for t in range(steps):
        z = pre[t * batch : (t + 1) * batch] + h @ w
        i, f, g, o = sigmoid(z[:, :hidden]), sigmoid(z[:, hidden : 2 * hidden]), np.tanh(z[:, 2 * hidden : 3 * hidden]), sigmoid(z[:, 3 * hidden :])
        kept.append((i, f, g, o, c))
        c = f * c + i * g
        h = o * np.tanh(c)
        kept[-1] += (np.tanh(c),)
        hs.append(h)
    dh, dc, dz = np.zeros_like(h), np.zeros_like(h), [None] * steps
    for t in reversed(range(steps)):
        i, f, g, o, before, tc = kept[t]
        d = dh + dh_all[t * batch : (t + 1) * batch]
        dc = dc + d * o * (1 - tc * tc)
        dz[t] = np.concatenate([dc * g * i * (1 - i), dc * before * f * (1 - f), dc * i * (1 - g * g), d * tc * o * (1 - o)], 1)
        dc = dc * f
        dh = dz[t] @ w.T
    return np.concatenate(hs), np.concatenate(dz), dh, dc


@pytest.mark.parametrize("initial", [False, True])
@pytest.mark.parametrize("steps,batch,hidden", SIZES)
def test_sequence_and_gradient(capi, steps, batch, hidden, initial):
    r = rng(steps * 7 + batch + hidden)
    ld = 4 * hidden + 4 * initial
    pre = r.standard_normal((steps * batch, 4 * hidden)).astype(np.float32)
    w = (r.uniform(-1, 1, (hidden, ld)) / np.sqrt(hidden)).astype(np.float32)
    h0, c0 = (r.uniform(-1, 1, (batch, hidden)).astype(np.float32) * initial for _ in range(2))
    dh = r.standard_normal((steps * batch, hidden)).astype(np.float32)
    want = reference(pre, w[:, : 4 * hidden], h0, c0, dh, steps, batch, hidden)
    d = [capi.to_device(v) for v in (pre, w, h0, c0, dh)]
    h, saved, dgates, dh0, dc0 = (capi.empty(s) for s in ((steps * batch, hidden), (6, steps * batch, hidden), (steps * batch, 4 * hidden),
                                                            (batch, hidden), (batch, hidden)))
    sizes = (i64(steps), i64(batch), i64(hidden))
    state = (d[2].ptr, d[3].ptr) if initial else (None, None)
    for _ in range(2):  # the second time in memory that the first has used
        capi.call("lstm_sequence", d[0].ptr, d[1].ptr, i64(ld), *state, *sizes, saved.ptr, h.ptr)
        capi.call("lstm_sequence_backward", saved.ptr, d[1].ptr, i64(ld), state[1], d[4].ptr, *sizes, dgates.ptr, dh0.ptr if initial else None,
                  dc0.ptr if initial else None)
    code = C.c_int(0)
    capi.call("device_status", C.byref(code))
    assert code.value == 0
    got = [h.numpy(), dgates.numpy()] + ([dh0.numpy(), dc0.numpy()] if initial else [])
    # fp32 sums of `hidden` terms per timestep (4 hidden in the gradient), carried through at most `steps` contracting timesteps
    bound = 2.0**-24 * (20 + 2 * np.sqrt(hidden)) * steps
    for a, b in zip(got, want):
        assert np.max(np.abs(a - b)) <= bound * max(1.0, np.abs(b).max())


def test_nan_travels_like_a_value(capi):
    """An output that is NaN goes from block to block as a code; its row is NaN from then on, the others are what they are without it."""
    steps, batch, hidden = 6, 18, 40
    r = rng(5)
    pre = r.standard_normal((steps, batch, 4 * hidden)).astype(np.float32)
    w = (r.uniform(-1, 1, (hidden, 4 * hidden)) / np.sqrt(hidden)).astype(np.float32)
    got = []
    for bad in (False, True):
        if bad:
            pre[1, 17, 3] = np.nan
        p, d = capi.to_device(pre), capi.to_device(w)
        h, saved = capi.empty((steps, batch, hidden)), capi.empty((6, steps * batch, hidden))
        capi.call("lstm_sequence", p.ptr, d.ptr, i64(4 * hidden), None, None, i64(steps), i64(batch), i64(hidden), saved.ptr, h.ptr)
        got.append(h.numpy())
    assert np.isnan(got[1][2:, 17]).all() and np.isnan(got[1][1, 17, 3]) and np.isnan(got[1][1]).sum() == 1
    assert np.array_equal(got[0][:, :17], got[1][:, :17]) and np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("batch,hidden", [(20, 40), (64, 512)])
def test_a_wait_that_runs_out_is_reported(batch, hidden, backward):
    """Blocks that do not wait for one another at all: the kernel ends, the next synchronising call says so, and the calls after it are right."""
    api, steps, r = rusttensor_b200.CApi(), 4, rng(batch)
    pre, dh = (r.standard_normal((steps * batch, c * hidden)).astype(np.float32) for c in (4, 1))
    w, zero = (r.uniform(-1, 1, (hidden, 4 * hidden)) / np.sqrt(hidden)).astype(np.float32), np.zeros((batch, hidden), np.float32)
    d = [api.to_device(v) for v in (pre, w, dh)]
    h, saved, dgates = (api.empty(s) for s in ((steps * batch, hidden), (6, steps * batch, hidden), (steps * batch, 4 * hidden)))
    sizes = (i64(steps), i64(batch), i64(hidden))

    def forward():
        api.call("lstm_sequence", d[0].ptr, d[1].ptr, i64(4 * hidden), None, None, *sizes, saved.ptr, h.ptr)

    def gradient():
        api.call("lstm_sequence_backward", saved.ptr, d[1].ptr, i64(4 * hidden), None, d[2].ptr, *sizes, dgates.ptr, None, None)

    forward()
    api.call("lstm_sequence_polls", i64(0))
    gradient() if backward else forward()
    code = C.c_int(0)
    with pytest.raises(Exception, match="gave up"):
        api.call("device_status", C.byref(code))
    assert code.value == 81
    api.call("device_status", C.byref(code))
    assert code.value == 0
    api.call("lstm_sequence_polls", i64(-1))
    forward()
    gradient()
    want = reference(pre, w, zero, zero, dh, steps, batch, hidden)
    for a, b in zip((h.numpy(), dgates.numpy()), want):
        assert np.max(np.abs(a - b)) <= 2.0**-24 * (20 + 2 * np.sqrt(hidden)) * steps * max(1.0, np.abs(b).max())
    api.close()


def test_sizes_are_checked(capi):
    x = capi.empty((4, 16))
    for sizes in ((0, 2, 4), (1, 0, 4), (1, 2, 0)):
        with pytest.raises(Exception, match="extents must be positive"):
            capi.call("lstm_sequence", x.ptr, x.ptr, i64(16), None, None, *[i64(s) for s in sizes], x.ptr, x.ptr)
    with pytest.raises(Exception, match="leading dimension"):
        capi.call("lstm_sequence", x.ptr, x.ptr, i64(15), None, None, i64(1), i64(2), i64(4), x.ptr, x.ptr)


@pytest.mark.parametrize("vocab,hidden,steps,batch", [(7, 9, 2, 3), (65, 24, 2, 17), (30, 200, 33, 16), (50, 130, 5, 40), (12, 64, 140, 4), (20, 512, 3, 90)])
def test_cells_written_op_by_op_become_a_sequence_in_a_capture(capi, vocab, hidden, steps, batch):
    dims = [vocab, hidden, steps, batch]
    params, inputs = workload_data(5, dims, seed=steps)
    results, launches = [], []
    for mode in ("step_eager", "step"):
        tr = rusttensor_b200.DataParallelTrainer(5, dims)
        for t, p in zip(tr.params, params):
            t.update_from_host(p)
        before = capi.launches()
        for _ in range(2):
            getattr(tr, mode)(inputs)
        launches.append(capi.launches() - before)
        results.append([p.numpy() for p in tr.params] + [tr.state(0, i).numpy() for i in range(len(params))] + [np.array(tr.last_loss())])
    if steps > 10:
        assert launches[1] < 2 * steps < launches[0]
    for a, b in zip(*results):  # two orders of the same fp32 sums, an Adam step of 1e-3 behind them
        assert_close(b, a, 1e-4, "captured and eager", abs_floor=5e-7)
