"""Elementwise programs that are reduced in the same launch (column sums of a bias gradient's term, the logsumexp of a row) against float64,
through the front end: rows and columns at the edges of the kernels' tiles, of vectors of four and of the longest row they take."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (3, 4), (5, 31), (33, 57), (16, 128), (17, 129), (64, 1000), (130, 1025), (1100, 1000), (1025, 1027), (3, 8192), (3, 8193), (2, 8200)]


@pytest.mark.parametrize("rows,cols", SHAPES)
def test_chain_with_both_reductions(gpu_engine, rows, cols):
    e, o = gpu_engine, gpu_engine.ops
    r = np.random.default_rng(rows + cols)
    xv, bv = r.standard_normal((rows, cols)).astype(np.float32), r.standard_normal(cols).astype(np.float32)
    if rows > 2:
        xv[1] += 90  # a row whose logsumexp lies far from the others
    x, b = e.tensor(xv, requires_grad=True), e.tensor(bv, requires_grad=True)
    sq = o.square(x)
    y = o.add(o.add(o.tanh(o.mul(x, b)), o.exp(o.mul_scalar(sq, -1.0))), o.div(o.sin(x), o.add(sq, e.tensor(np.float32(1).reshape(())))))
    lse = o.logsumexp(y, 1)
    o.sum(lse).backward()
    X, B = xv.astype(np.float64), bv.astype(np.float64)
    t, q = np.tanh(X * B), 1 + X * X
    Y = t + np.exp(-X * X) + np.sin(X) / q
    m = Y.max(1, keepdims=True)
    L = m + np.log(np.exp(Y - m).sum(1, keepdims=True))
    dy = np.exp(Y - L)
    dt = dy * (1 - t * t)
    dx = dt * B + dy * (np.cos(X) / q - 2 * X * np.exp(-X * X) - 2 * X * np.sin(X) / q**2)
    # a handful of fp32 operations of order one an element, a sum of `cols` or `rows` terms behind them
    np.testing.assert_allclose(lse.numpy(), L[:, 0], rtol=2e-6, atol=2e-6)
    assert np.abs(x.grad.numpy() - dx).max() <= 4e-6 * max(1.0, np.abs(dx).max())
    assert np.abs(b.grad.numpy() - (dt * X).sum(0)).max() <= 4e-6 * max(1.0, np.abs(dt * X).sum(0).max())


@pytest.mark.parametrize("shape,axis", [((7, 1), 0), ((1, 7), 1), ((1, 7), 0), ((1, 7), None), ((5, 6), 0), ((5, 6), None)], ids=str)
def test_the_chain_over_other_axes(gpu_engine, shape, axis):
    # 2-D expressions whose reduction is not over their rows, and the ones where the two coincide
    e, o = gpu_engine, gpu_engine.ops
    xv = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    x, b = e.tensor(xv, requires_grad=True), e.tensor(np.full(shape[1], 0.5, np.float32))
    sq = o.square(x)
    y = o.add(o.add(o.tanh(o.mul(x, b)), o.exp(o.mul_scalar(sq, -1.0))), o.div(o.sin(x), o.add(sq, e.tensor(np.float32(1).reshape(())))))
    lse = o.logsumexp(y, axis)
    o.sum(lse).backward()
    X = xv.astype(np.float64)
    t, q = np.tanh(X / 2), 1 + X * X
    Y = t + np.exp(-X * X) + np.sin(X) / q
    L = np.log(np.exp(Y).sum(axis, keepdims=True))
    dx = np.exp(Y - L) * ((1 - t * t) / 2 + np.cos(X) / q - 2 * X * np.exp(-X * X) - 2 * X * np.sin(X) / q**2)
    np.testing.assert_allclose(lse.numpy().reshape(-1), L.reshape(-1), rtol=2e-6, atol=2e-6)
    assert np.abs(x.grad.numpy() - dx).max() <= 4e-6 * max(1.0, np.abs(dx).max())


def special_rows(rows, cols):
    x = np.random.default_rng(rows + cols).standard_normal((rows, cols)).astype(np.float32)
    x[1], x[2, 3], x[3, 1], x[4, 0], x[5] = -np.inf, -np.inf, np.inf, np.nan, np.inf
    x[6, 0], x[6, 1], x[7, 2], x[7, 3] = np.inf, -np.inf, np.inf, np.nan
    return x


@pytest.mark.parametrize("rows,cols", [(8, 9), (20, 128), (9, 1030)])
@pytest.mark.parametrize("chain", ["alone", "scaled", "workload"])
def test_rows_of_infinities_and_nan(gpu_engine, rows, cols, chain):
    """Row by row what the reference gives, also through the gradient, which is elementwise in the forward result: an infinity of either sign that is the
    largest of its row, one that is not, NaN, and rows beside them."""
    xv, out = special_rows(rows, cols), []
    for e in (gpu_engine, oracle.engine()):
        o = e.ops
        x, b = e.tensor(xv, requires_grad=True), e.tensor(np.full(cols, 0.5, np.float32), requires_grad=True)
        if chain == "workload":  # the program that logsumexp_kernel carries; the sine of an infinity is NaN
            sq = o.square(x)
            y = o.add(o.add(o.tanh(o.mul(x, b)), o.exp(o.mul_scalar(sq, -1.0))), o.div(o.sin(x), o.add(sq, e.tensor(np.float32(1).reshape(())))))
        else:
            y = o.mul_scalar(x, 0.5) if chain == "scaled" else x
        lse = o.logsumexp(y, 1)
        o.sum(lse).backward()
        out.append([lse.numpy(), x.grad.numpy()])
    for got, want in zip(*out):
        # exp and its sum to a few units in the last place of values of order one
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=2e-6)
