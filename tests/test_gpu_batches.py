"""Inputs of a step: several parts of one upload, rows of several matrices gathered by uploaded numbers, concatenation of many pieces,
sums of several matrices' columns; and the optimizer's launch that advances the step count."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from rusttensor_b200 import CApi

    a = CApi()
    yield a
    a.close()


@pytest.mark.parametrize("parts", [1, 2, 9])  # the kernel copies eight at a time
def test_upload_parts(api, parts):
    r = np.random.default_rng(parts)
    sizes = [1 + 37 * i for i in range(parts)]
    at = np.cumsum([0] + [(4 * n + 255) // 256 * 256 for n in sizes])
    for _ in range(2):  # the second upload takes over what the first has left
        up, dst = C.c_void_p(), [api.to_device(np.zeros(n, np.float32)) for n in sizes]
        api.call("upload_create", C.c_size_t(int(at[-1])), C.byref(up))
        offsets, nbytes = (C.c_int64 * parts)(*at[:-1].tolist()), (C.c_int64 * parts)(*[4 * n for n in sizes])
        ptrs = (C.c_void_p * parts)(*[d.ptr.value for d in dst])
        for _ in range(3):
            p, data = C.c_void_p(), [r.random(n, dtype=np.float32) for n in sizes]
            api.call("upload_host_buffer", up, C.byref(p))
            for a, o in zip(data, at):
                C.memmove(p.value + int(o), a.ctypes.data, a.nbytes)
            api.call("upload_submit_parts", up, parts, offsets, nbytes, ptrs)
            for a, d in zip(data, dst):
                np.testing.assert_array_equal(a, d.numpy())
        nbytes[0] = int(at[-1]) + 1
        with pytest.raises(Exception, match="ends behind"):
            api.call("upload_submit_parts", up, parts, offsets, nbytes, ptrs)
        api.call("upload_destroy", up)


@pytest.mark.parametrize("n_idx", [1, 7, 301, 5000])  # one to eight rows a block, the last of them not full
def test_gather_rows_list(api, n_idx):
    r = np.random.default_rng(n_idx)
    rows, lens = 613, [1, 10, 784, 0]
    data = [r.random((rows, n), dtype=np.float32) for n in lens]
    src, dst = [api.to_device(d) for d in data[:3]], [api.to_device(np.ones((n_idx, n), np.float32)) for n in lens[:3]]
    up, p = C.c_void_p(), C.c_void_p()
    api.call("upload_create", C.c_size_t(4 * n_idx), C.byref(up))
    ptrs = lambda ts: (C.c_void_p * 4)(*[t.ptr.value for t in ts], None)  # noqa: E731
    for _ in range(3):
        api.call("upload_host_buffer", up, C.byref(p))
        idx = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_int32)), (n_idx,))
        idx[:] = r.integers(0, rows, n_idx)
        want = [d[idx] for d in data]
        idx[-1] = rows  # outside: a row of zeros
        api.call("upload_gather_rows", up, 4, ptrs(src), (C.c_int64 * 4)(*lens), C.c_int64(rows), C.c_int64(n_idx), ptrs(dst))
        for w, d in zip(want, dst):
            w[-1] = 0
            np.testing.assert_array_equal(w, d.numpy())
    api.call("upload_destroy", up)


@pytest.mark.parametrize("n_src", [8, 9, 17])  # a launch takes eight; one of them is empty
def test_gather_rows_of_many_matrices(api, n_src):
    r = np.random.default_rng(n_src)
    rows, n_idx, lens = 61, 40, [(3 * i) % 29 for i in range(n_src)]
    data, pick = [r.random((rows, n), dtype=np.float32) for n in lens], r.integers(0, rows, n_idx)
    src, dst = [api.to_device(d) if d.size else None for d in data], [api.to_device(np.ones((n_idx, n), np.float32)) if n else None for n in lens]
    up, p = C.c_void_p(), C.c_void_p()
    api.call("upload_create", C.c_size_t(4 * n_idx), C.byref(up))
    api.call("upload_host_buffer", up, C.byref(p))
    np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_int32)), (n_idx,))[:] = pick
    ptrs = lambda ts: (C.c_void_p * n_src)(*[t.ptr.value if t else None for t in ts])  # noqa: E731
    api.call("upload_gather_rows", up, n_src, ptrs(src), (C.c_int64 * n_src)(*lens), C.c_int64(rows), C.c_int64(n_idx), ptrs(dst))
    for d, o in zip(data, dst):
        if o:
            np.testing.assert_array_equal(d[pick], o.numpy())
    api.call("upload_destroy", up)


@pytest.mark.parametrize("outer,lens", [(1, [5]), (1, [4] * 300), (7, [3, 0, 8, 129]), (3, [4, 2000, 16])])  # more pieces than a launch takes
def test_concat_list(api, outer, lens):
    r = np.random.default_rng(len(lens))
    data = [r.random((outer, n), dtype=np.float32) for n in lens]
    src, out = [api.to_device(d) if d.size else None for d in data], api.to_device(np.zeros((outer, sum(lens)), np.float32))
    ptrs = (C.c_void_p * len(lens))(*[s.ptr.value if s else None for s in src])
    api.call("concat_list", len(lens), ptrs, (C.c_int64 * len(lens))(*lens), C.c_int64(outer), out.ptr)
    np.testing.assert_array_equal(out.numpy(), np.concatenate(data, 1))


@pytest.mark.parametrize("shapes", [[(1, 1)], [(31, 33), (513, 32), (0, 5), (2048, 7)], [(64, 10 + i) for i in range(35)]])  # more than a launch takes
def test_column_sums_list(api, shapes):
    r = np.random.default_rng(len(shapes))
    data = [r.random(s, dtype=np.float32) for s in shapes]
    src, out = [api.to_device(d) if d.size else None for d in data], [api.to_device(np.ones(s[1], np.float32)) for s in shapes]
    n = len(shapes)
    api.call("column_sums_list", n, (C.c_void_p * n)(*[s.ptr.value if s else None for s in src]), (C.c_int64 * n)(*[s[0] for s in shapes]),
             (C.c_int64 * n)(*[s[1] for s in shapes]), (C.c_void_p * n)(*[o.ptr.value for o in out]))
    for d, o in zip(data, out):
        np.testing.assert_allclose(o.numpy(), d.sum(0, dtype=np.float64), rtol=1e-6)


@pytest.mark.parametrize("tensors", [1, 3, 200])  # one block; several; more tensors than a launch takes
@pytest.mark.parametrize("kind", [1, 2])
def test_optimizer_step_counts_itself(api, kind, tensors):
    r = np.random.default_rng(tensors)
    sizes = [int(n) for n in r.integers(1, 3000, tensors)]
    new = lambda: [r.standard_normal(n).astype(np.float32) for n in sizes]  # noqa: E731
    p, g, s1, s2 = new(), new(), new(), [x * x for x in new()]
    f = C.c_float
    got = []
    for name in ("device_t", "next"):
        dev = [[api.to_device(x) for x in xs] for xs in (p, g, s1, s2)]
        lists = [(C.c_void_p * tensors)(*[d.ptr.value for d in ds]) for ds in dev]
        state = api.to_device(np.array([0, 0, 7, 0], np.int32).view(np.float32))
        for _ in range(3):
            if name == "device_t":
                api.call("dp_step_begin", state.ptr)
            api.call("optimizer_step_multi_" + name, kind, tensors, *lists, (C.c_int64 * tensors)(*sizes), f(1e-2), f(0.9), f(0.999), f(1e-8), f(0.9),
                     state.ptr, f(1.0), 0, f(0), f(0))
        assert state.numpy().view(np.int32).tolist() == [3, 0, 10, 0]
        got.append([d.numpy() for ds in dev for d in ds])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
