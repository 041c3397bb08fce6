"""Convolutions of the TMA-fed tensor-core kernel against float64: extents that its pixel boxes and 32-channel blocks do not divide,
strides, output phases, one and several column tiles."""
import ctypes as C

import numpy as np
import pytest

import ref_f64

pytestmark = pytest.mark.gpu

i64 = C.c_int64
CASES = [(64, 33, 30, 30, 70, 3, 1, 1), (90, 48, 29, 37, 96, 5, 2, 2), (24, 16, 41, 33, 16, 3, 1, 0), (40, 130, 23, 31, 130, 1, 1, 0),
         (48, 20, 50, 46, 65, 4, 2, 1), (16, 17, 64, 67, 24, 3, 3, 1)]


@pytest.fixture(scope="module")
def api():
    from rusttensor_b200 import CApi

    a = CApi()
    yield a
    a.close()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,cin,h,w,cout,k,s,p", CASES)
def test_convolution(api, n, cin, h, w, cout, k, s, p, transposed):
    r = np.random.default_rng(n + cin + h)
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = r.standard_normal((cin, cout, k, k) if transposed else (cout, cin, k, k)).astype(np.float32)
    b = r.standard_normal(cout).astype(np.float32)
    some = [0, n // 2, n - 1]  # images that are checked (the reference takes its time)
    name, fwd, bwd = (("conv2d_transpose", ref_f64.conv2d_transpose, ref_f64.conv2d_transpose_backward) if transposed
                      else ("conv2d", ref_f64.conv2d, ref_f64.conv2d_backward))
    ref = fwd(x[some], wt, b, (s, s), (p, p))
    y, dx = api.empty((n,) + ref.shape[1:]), api.empty(x.shape)
    g = r.standard_normal(y.shape).astype(np.float32)
    dev = [api.to_device(v) for v in (x, wt, b, g)]
    dims = (i64(n), i64(cin), i64(h), i64(w), i64(cout), k, k, s, s, p, p)
    api.call(name, dev[0].ptr, dev[1].ptr, dev[2].ptr, *dims, y.ptr)
    api.call(name + "_backward", dev[0].ptr, dev[1].ptr, dev[3].ptr, *dims, dx.ptr, None, None)
    for got, want in ((y.numpy()[some], ref), (dx.numpy()[some], bwd(x[some], wt, g[some], (s, s), (p, p))[0])):
        assert np.all(np.abs(got - want) <= 4e-6 * np.abs(want).max() + 1e-6 * np.abs(want))


# The 16-bit parts (k_conv_parts.cu): from 2^30 multiply-adds on, both gradients from 2^31 (strided) and 2^32.  Channels that leave K-blocks and
# column tiles ragged, boxes that overhang, odd output extents of a stride of two, and inputs that need three parts.
PARTS = [(65, 70, 29, 31, 66, 3, 1, 1), (130, 40, 40, 38, 84, 3, 1, 1), (96, 33, 37, 35, 97, 4, 2, 1), (70, 66, 33, 30, 68, 5, 2, 2)]


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,cin,h,w,cout,k,s,p", PARTS)
def test_convolution_of_parts(api, n, cin, h, w, cout, k, s, p, transposed, spread):
    r = np.random.default_rng(n + cin + h)
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    if spread:  # one channel far below the others
        x[:, cin // 2] *= np.float32(2.0**-30)
    wt = (r.standard_normal((cin, cout, k, k) if transposed else (cout, cin, k, k)) / k).astype(np.float32)
    b = r.standard_normal(cout).astype(np.float32)
    some = [0, n // 2, n - 1]
    name, fwd, bwd = (("conv2d_transpose", ref_f64.conv2d_transpose, ref_f64.conv2d_transpose_backward) if transposed
                      else ("conv2d", ref_f64.conv2d, ref_f64.conv2d_backward))
    ref = fwd(x[some], wt, b, (s, s), (p, p))
    y, dx, dw, db = api.empty((n,) + ref.shape[1:]), api.empty(x.shape), api.empty(wt.shape), api.empty(b.shape)
    g = np.zeros(y.shape, np.float32)  # the weight gradient is checked too: upstream gradient in the images that the reference looks at
    g[some] = r.standard_normal((3,) + y.shape[1:]).astype(np.float32)
    dev = [api.to_device(v) for v in (x, wt, b, g)]
    dims = (i64(n), i64(cin), i64(h), i64(w), i64(cout), k, k, s, s, p, p)
    api.call(name, dev[0].ptr, dev[1].ptr, dev[2].ptr, *dims, y.ptr)
    api.call(name + "_backward", dev[0].ptr, dev[1].ptr, dev[3].ptr, *dims, dx.ptr, dw.ptr, db.ptr)
    want = bwd(x[some], wt, g[some], (s, s), (p, p))
    rows, cols = cin * k * k, y.shape[2] * y.shape[3] * 3
    # relative to the root of the number of terms: 32 additions with truncation between roundings, the parts' own 2^-22
    for got, ref_, terms in ((y.numpy()[some], ref, rows), (dx.numpy()[some], want[0], cout * k * k), (dw.numpy(), want[1], cols), (db.numpy(), want[2], cols)):
        assert np.abs(got - ref_).max() <= (32 * 2.0**-23 + 2.0**-21) * (np.abs(ref_).max() + np.sqrt(terms))
    if spread and not transposed:  # the small channel's weight gradient has its own scale
        small, ref_ = dw.numpy()[:, cin // 2], want[1][:, cin // 2]
        assert np.abs(small - ref_).max() <= 4e-6 * np.abs(ref_).max() + 1e-6 * np.abs(ref_).max()


@pytest.mark.parametrize("octaves", [28, 31, 40])
def test_convolution_of_parts_of_wide_ranges(api, octaves):
    """Magnitudes spread over so many powers of two in every channel and filter, and results whose terms all weigh the same: what the small elements
    keep shows."""
    n, cin, h, w, cout = 65, 70, 28, 32, 128  # no short segments at the ends, which would be told from their largest element
    r = np.random.default_rng(octaves)

    def spread(*shape):
        return (np.exp2(r.uniform(-octaves / 2, octaves / 2, shape)) * r.choice([-1, 1], shape)).astype(np.float32)

    x, g, wt = spread(n, cin, h, w), spread(n, cout, h, w), spread(cout, cin, 3, 3)
    g[:, 2] = 1 / np.abs(x[:, 1])                                   # the weight gradient of channels 1 -> 2, middle tap
    wt[:, 3] = 1 / np.abs(g[4, :, 9:12, 11:14])[:, ::-1, ::-1]      # the input gradient of image 4, channel 3, pixel (10, 12)
    wt[0] = 1 / np.abs(x[3, :, 9:12, 11:14])                        # the output of image 3, channel 0, pixel (10, 12)
    y, dx, dw, db = api.empty(g.shape), api.empty(x.shape), api.empty(wt.shape), api.empty((cout,))
    dev = [api.to_device(v) for v in (x, wt, np.zeros(cout, np.float32), g)]
    dims = (i64(n), i64(cin), i64(h), i64(w), i64(cout), 3, 3, 1, 1, 1, 1)
    api.call("conv2d", dev[0].ptr, dev[1].ptr, dev[2].ptr, *dims, y.ptr)
    api.call("conv2d_backward", dev[0].ptr, dev[1].ptr, dev[3].ptr, *dims, dx.ptr, dw.ptr, db.ptr)
    for got, a, b in ((y.numpy()[3, 0, 10, 12], x[3, :, 9:12, 11:14], wt[0]), (dx.numpy()[4, 3, 10, 12], g[4, :, 9:12, 11:14], wt[:, 3, ::-1, ::-1]),
                      (dw.numpy()[2, 1, 1, 1], g[:, 2], x[:, 1])):
        terms = a.astype(np.float64) * b
        # 32 additions with truncation between two roundings, the parts' own 2^-22
        assert abs(got - terms.sum()) <= (32 * 2.0**-23 + 2.0**-21) * np.abs(terms).sum()


@pytest.mark.parametrize("power", [-34, -30, -26, -18])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("h,w", [(64, 64), (61, 67)])
def test_pixels_far_below_the_rest(api, h, w, transposed, power):
    """Of which the outputs at the same places are made, all channels of them: too few to be counted."""
    n, cin, cout = 128, 32, 128
    at = (3, 10, 11), (n - 1, h - 1, w - 1)
    r = np.random.default_rng(h - power)
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = r.standard_normal((cin, cout, 1, 1) if transposed else (cout, cin, 1, 1)).astype(np.float32)
    for i, v, u in at:
        x[i, :, v, u] *= np.float32(2.0**power)
    y = api.empty((n, cout, h, w))
    dev = [api.to_device(v) for v in (x, wt, np.zeros(cout, np.float32))]
    api.call("conv2d_transpose" if transposed else "conv2d", *[d.ptr for d in dev], i64(n), i64(cin), i64(h), i64(w), i64(cout), 1, 1, 1, 1, 0, 0, y.ptr)
    got, m = y.numpy(), wt[:, :, 0, 0].astype(np.float64).T if transposed else wt[:, :, 0, 0].astype(np.float64)
    for i, v, u in at:
        p = x[i, :, v, u].astype(np.float64)
        # the parts' own 2^-21, four additions with truncation
        assert np.all(np.abs(got[i, :, v, u] - m @ p) <= (2.0**-21 + 4 * 2.0**-23) * (np.abs(m) @ np.abs(p)))


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,cin,h,w,cout,k,s,p", [(65, 70, 29, 31, 66, 3, 1, 1), (96, 33, 37, 35, 97, 4, 2, 1), (70, 66, 33, 30, 68, 5, 2, 2)])
def test_infinities_and_nan_stay_where_they_belong(api, n, cin, h, w, cout, k, s, p, transposed):
    """An infinity or NaN in the input (the upstream gradient) shows in the outputs that it is a term of, and in no others."""
    r = np.random.default_rng(n)
    name, fwd, bwd = (("conv2d_transpose", ref_f64.conv2d_transpose, ref_f64.conv2d_transpose_backward) if transposed
                      else ("conv2d", ref_f64.conv2d, ref_f64.conv2d_backward))
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = (r.standard_normal((cin, cout, k, k) if transposed else (cout, cin, k, k)) / k).astype(np.float32)
    b, some = r.standard_normal(cout).astype(np.float32), [1, n - 1]
    clean = fwd(x[some], wt, b, (s, s), (p, p))
    y, dx = api.empty((n,) + clean.shape[1:]), api.empty(x.shape)
    g = r.standard_normal(y.shape).astype(np.float32)

    def spoil(a):
        a[some[0], 3, a.shape[2] // 2, 4], a[some[0], 5, 2, a.shape[3] - 2], a[some[1], 0, 0, 0] = np.inf, np.nan, -np.inf
        return a

    # which elements a spoiled one is a term of: those that change with it
    def touched(f, a):
        zero = np.zeros_like(a[some])
        return f(np.where(np.isfinite(a[some]), zero, 1.0)) != 0

    def run():
        dev = [api.to_device(v) for v in (x, wt, b, g)]
        dims = (i64(n), i64(cin), i64(h), i64(w), i64(cout), k, k, s, s, p, p)
        api.call(name, dev[0].ptr, dev[1].ptr, dev[2].ptr, *dims, y.ptr)
        api.call(name + "_backward", dev[0].ptr, dev[1].ptr, dev[3].ptr, *dims, dx.ptr, None, None)
        return y.numpy()[some], dx.numpy()[some]

    before = run()
    spoil(x), spoil(g)
    after = run()
    positive = np.abs(wt)
    for was, now, hit in ((before[0], after[0], touched(lambda v: fwd(v, positive, None, (s, s), (p, p)), x)),
                          (before[1], after[1], touched(lambda v: bwd(np.ones_like(x[some]), positive, v, (s, s), (p, p))[0], g))):
        assert not np.isfinite(now[hit]).any()
        assert np.isfinite(now[~hit]).all() and np.abs(now - was)[~hit].max() <= 1e-5 * np.abs(was).max()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,cin,h,w,cout,k,s,p", [(130, 40, 40, 38, 84, 3, 1, 1), (96, 33, 37, 35, 97, 4, 2, 1), (70, 66, 33, 30, 68, 5, 2, 2)])
def test_infinities_and_nan_in_weight_gradients(api, n, cin, h, w, cout, k, s, p, transposed):
    """Of the wide side (the input, the upstream gradient of a transposed convolution), whose elements meet the padding of the other side's boxes."""
    r = np.random.default_rng(n)
    name, bwd = ("conv2d_transpose", ref_f64.conv2d_transpose_backward) if transposed else ("conv2d", ref_f64.conv2d_backward)
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = (r.standard_normal((cin, cout, k, k) if transposed else (cout, cin, k, k)) / k).astype(np.float32)
    side = (lambda v: (v - 1) * s + k - 2 * p) if transposed else (lambda v: (v + 2 * p - k) // s + 1)
    g = r.standard_normal((n, cout, side(h), side(w))).astype(np.float32)
    some, wide = [1, n - 1], g if transposed else x

    def run():
        dev = [api.to_device(v) for v in (x, wt, g)]
        dx, dw, db = api.empty(x.shape), api.empty(wt.shape), api.empty((cout,))
        api.call(name + "_backward", *[d.ptr for d in dev], i64(n), i64(cin), i64(h), i64(w), i64(cout), k, k, s, s, p, p, dx.ptr, dw.ptr, db.ptr)
        return dw.numpy()

    was = run()
    wide[1, 3, wide.shape[2] // 2, 4], wide[1, 5, 2, -1], wide[n - 1, 0, -1, 7], wide[n - 1, 7, 0, 0] = np.inf, np.nan, -np.inf, np.inf
    marks = np.where(np.isfinite(wide[some]), 0.0, 1.0)
    hit = (bwd(np.ones_like(x[some]), wt, marks, (s, s), (p, p)) if transposed else bwd(marks, wt, np.ones_like(g[some]), (s, s), (p, p)))[1] != 0
    now = run()
    assert not np.isfinite(now[hit]).any() and np.isfinite(now[~hit]).all()
    # 32 additions with truncation between roundings, the parts' own 2^-22, on either side
    assert np.abs(now - was)[~hit].max() <= 2 * (32 * 2.0**-23 + 2.0**-21) * (np.abs(was).max() + np.sqrt(n * side(h) * side(w)))


# Kernels, strides and paddings that differ between the dimensions, strides of three and eight, padding of the kernel's size and more (work as above).
FORMS = [(64, 48, 40, 44, 80, (3, 5), (1, 1), (1, 2)), (64, 64, 40, 48, 96, (5, 3), (1, 2), (2, 1)), (128, 64, 60, 63, 80, (3, 3), (3, 3), (1, 1)),
         (128, 70, 96, 90, 80, (4, 5), (8, 7), (0, 2)), (104, 48, 28, 28, 80, (3, 3), (1, 1), (4, 5)), (96, 64, 30, 32, 72, (4, 3), (2, 2), (5, 3))]


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,cin,h,w,cout,k,s,p", FORMS)
def test_forms_of_convolutions_of_parts(api, n, cin, h, w, cout, k, s, p, transposed):
    r = np.random.default_rng(n + cin + h)
    if transposed and s[0] > 2:
        h, w = h // s[0], w // s[1]
    x = r.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = (r.standard_normal((cin, cout, *k) if transposed else (cout, cin, *k)) / k[0]).astype(np.float32)
    b = r.standard_normal(cout).astype(np.float32)
    some = [0, n - 1]
    name, fwd, bwd = (("conv2d_transpose", ref_f64.conv2d_transpose, ref_f64.conv2d_transpose_backward) if transposed
                      else ("conv2d", ref_f64.conv2d, ref_f64.conv2d_backward))
    ref = fwd(x[some], wt, b, s, p)
    y, dx, dw, db = api.empty((n,) + ref.shape[1:]), api.empty(x.shape), api.empty(wt.shape), api.empty(b.shape)
    g = np.zeros(y.shape, np.float32)
    g[some] = r.standard_normal((2,) + y.shape[1:]).astype(np.float32)
    dev = [api.to_device(v) for v in (x, wt, b, g)]
    dims = (i64(n), i64(cin), i64(h), i64(w), i64(cout), *k, *s, *p)
    api.call(name, dev[0].ptr, dev[1].ptr, dev[2].ptr, *dims, y.ptr)
    api.call(name + "_backward", dev[0].ptr, dev[1].ptr, dev[3].ptr, *dims, dx.ptr, dw.ptr, db.ptr)
    want = bwd(x[some], wt, g[some], s, p)
    taps = k[0] * k[1]
    for got, ref_, terms in ((y.numpy()[some], ref, cin * taps), (dx.numpy()[some], want[0], cout * taps), (dw.numpy(), want[1], 2 * y.shape[2] * y.shape[3]),
                             (db.numpy(), want[2], 2 * y.shape[2] * y.shape[3])):
        assert np.abs(got - ref_).max() <= (32 * 2.0**-23 + 2.0**-21) * (np.abs(ref_).max() + np.sqrt(terms))
