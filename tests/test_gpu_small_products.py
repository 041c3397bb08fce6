"""Small products (one launch: split reduction, bias, activation) and the list entries of recurrent layers against float64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

i64 = C.c_int64
# one element, edges of the 32 x 64 tile and of the 64-deep block of the reduction, cluster splits 1..8, rows that 128-bit loads
# cannot take, the largest products of this kernel's range
SIZES = [(1, 1, 1), (31, 63, 63), (32, 64, 64), (33, 65, 65), (5, 129, 700), (64, 577, 130), (200, 512, 66), (2, 4096, 3), (512, 64, 1000)]


@pytest.fixture(scope="module")
def api():
    from rusttensor_b200 import CApi

    a = CApi()
    yield a
    a.close()


def close(got, ref, scale):
    assert np.all(np.abs(got - ref) <= 3e-6 * scale + 1e-6 * np.abs(ref))


@pytest.mark.parametrize("m,k,n", SIZES)
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_small_product(api, m, k, n, trans):
    r = np.random.default_rng(m * 7 + k * 3 + n)
    a, b, c0 = (r.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    ta, tb = trans
    da, db = api.to_device(a.T if ta else a), api.to_device(b.T if tb else b)
    for accumulate in (0, 1):
        c = api.to_device(c0)
        api.call("gemm", ta, tb, i64(m), i64(n), i64(k), da.ptr, i64(m if ta else k), db.ptr, i64(k if tb else n), c.ptr, i64(n), accumulate)
        close(c.numpy(), a.astype(np.float64) @ b + accumulate * c0, np.sqrt(k))


# 128 x 64 tiles in one wave: one row and column more than a tile, a K-block and one, cluster splits 1 .. 16, partial sums in a workspace,
# copies of 4 and of 16 bytes; and the first size past one wave with a short reduction
@pytest.mark.parametrize("m,k,n", [(129, 321, 65), (128, 4100, 64), (37, 2049, 577), (300, 33, 2001), (96, 13000, 40), (1120, 144, 1748)])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_medium_product(api, m, k, n, trans):
    test_small_product(api, m, k, n, trans)


# one more than whole tiles and K-blocks, rows that TMA cannot fetch directly, 256- and 128-column tiles, chunks of 1, 2 and 4 K-blocks
@pytest.mark.parametrize("m,k,n", [(769, 65, 1025), (1024, 64, 768), (1030, 1024, 900), (6200, 100, 70), (2100, 2081, 1900)])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_large_product(api, m, k, n, trans):
    test_small_product(api, m, k, n, trans)


# up to 16 columns: blocks of 8 rows and chunks of 256 up to 16 rows an SM (2368 on 148), of 32 and 128 beyond
@pytest.mark.parametrize("m,k,n", [(7, 17, 1), (9, 255, 16), (8, 256, 3), (33, 257, 15), (2368, 513, 10), (2369, 129, 10), (4099, 300, 16)])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_product_of_few_columns(api, m, k, n, trans):
    test_small_product(api, m, k, n, trans)


@pytest.mark.parametrize("m,k,n", SIZES + [(300, 784, 300), (900, 70, 1000)])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_linear_layer(api, m, k, n, act):
    r = np.random.default_rng(m + k + n + act)
    a, b, bias = (r.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (n,)))
    f = [lambda v: v, lambda v: np.maximum(v, 0), np.tanh, lambda v: 1 / (1 + np.exp(-v))][act]
    ref = f(a.astype(np.float64) @ b + bias)
    da, db, dbias, c = api.to_device(a), api.to_device(b), api.to_device(bias), api.empty((m, n))
    api.call("gemm_bias_act", i64(m), i64(n), i64(k), da.ptr, i64(k), db.ptr, i64(n), dbias.ptr, act, c.ptr, i64(n))
    close(c.numpy(), ref, np.sqrt(k))
    many = [api.to_device(a[:, ::-1].copy()), da, da]
    outs = [api.empty((m, n)) for _ in many]
    P = C.c_void_p * len(many)
    api.call("gemm_bias_act_list", len(many), P(*[t.ptr for t in many]), P(*[t.ptr for t in outs]), i64(m), i64(n), i64(k), db.ptr, dbias.ptr, act)
    close(outs[0].numpy(), f(a[:, ::-1].astype(np.float64) @ b + bias), np.sqrt(k))
    for o in outs[1:]:
        close(o.numpy(), ref, np.sqrt(k))


@pytest.mark.parametrize("count,m,k,n", [(1, 3, 5, 7), (2, 64, 33, 65), (130, 8, 40, 36), (300, 5, 64, 20), (128, 64, 100, 256)])
def test_sums_over_uses_of_a_weight(api, count, m, k, n):
    r = np.random.default_rng(count + m + k + n)
    a, g = r.standard_normal((count, m, k)).astype(np.float32), r.standard_normal((count, m, n)).astype(np.float32)
    c0, b0 = r.standard_normal((k, n)).astype(np.float32), r.standard_normal(n).astype(np.float32)
    das, dgs = [api.to_device(x) for x in a], [api.to_device(x) for x in g]
    P = C.c_void_p * count
    c, b = api.to_device(c0), api.to_device(b0)
    api.call("gemm_sum_products", count, P(*[t.ptr for t in das]), P(*[t.ptr for t in dgs]), i64(m), i64(k), i64(n), c.ptr)
    close(c.numpy(), c0 + np.einsum("tmk,tmn->kn", a.astype(np.float64), g), np.sqrt(count * m))
    api.call("sum_rows_accumulate_list", count, P(*[t.ptr for t in dgs]), i64(m), i64(n), b.ptr)
    close(b.numpy(), b0 + g.astype(np.float64).sum((0, 1)), np.sqrt(count * m))
