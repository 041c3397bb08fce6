"""The tcgen05 3xTF32 tensor-core contractions against float64 and against the exact FP32 kernels.
3xTF32 keeps fp32-level accuracy (hi*hi + hi*lo + lo*hi with fp32 accumulation in tensor memory),
so the same 1e-4 bound as everywhere else applies; in practice the error is ~1e-6."""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_close, max_abs_rel, rng

pytestmark = pytest.mark.gpu


def gemm(capi, ta, tb, m, n, k, a, b, c0=None, accumulate=0, lda=None, ldb=None):
    da, db = capi.to_device(a), capi.to_device(b)
    dc = capi.to_device(c0) if c0 is not None else capi.empty((m, n))
    capi.call("gemm", C.c_int(ta), C.c_int(tb), C.c_int64(m), C.c_int64(n), C.c_int64(k), da.ptr, C.c_int64(lda or a.shape[1]),
              db.ptr, C.c_int64(ldb or b.shape[1]), dc.ptr, C.c_int64(n), C.c_int(accumulate))
    code = C.c_int(0)
    capi.call("device_status", C.byref(code))
    return dc.numpy()


SHAPES = [(128, 128, 32), (128, 128, 64), (256, 128, 3136), (256, 3136, 128), (3136, 128, 256), (64, 2048, 577), (577, 2048, 64),
          (64, 577, 2048), (130, 70, 33), (257, 129, 65), (1000, 24, 200), (128, 32, 4096), (512, 512, 512), (33, 17, 2000),
          # more 128x64 tiles than the GPU has multiprocessors: the shared-memory-operand kernel takes these
          (1024, 1536, 160), (2100, 1030, 72)]


@pytest.mark.parametrize("m,n,k", SHAPES, ids=str)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_tensor_core_gemm_matches_float64_and_fp32_path(capi, m, n, k, ta, tb):
    r = rng(m * 7 + n * 3 + k + ta * 2 + tb)
    a = r.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    b = r.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    A = (a.T if ta else a).astype(np.float64)
    B = (b.T if tb else b).astype(np.float64)
    ref = A @ B
    capi.call("set_tensor_cores", C.c_int(1))
    l0 = capi.launches()
    tc = gemm(capi, ta, tb, m, n, k, a, b)
    capi.call("set_tensor_cores", C.c_int(0))
    fp = gemm(capi, ta, tb, m, n, k, a, b)
    capi.call("set_tensor_cores", C.c_int(1))
    assert_close(tc, ref, 1e-4, "tensor-core gemm vs float64")
    assert_close(tc, fp, 1e-4, "tensor-core gemm vs FP32 kernel")
    # fp32-level accuracy: the error against float64 is of the same order as the exact-FP32 kernel's
    scale = np.abs(A) @ np.abs(B)
    e_tc = float(np.max(np.abs(tc - ref) / scale))
    e_fp = float(np.max(np.abs(fp - ref) / scale))
    assert e_tc < 4e-6, (e_tc, e_fp)


def test_tensor_core_gemm_accumulate_and_unaligned_ld(capi):
    r = rng(5)
    m, n, k = 256, 192, 100
    a = r.standard_normal((m, k + 1)).astype(np.float32)  # lda = k+1: rows are not 16-byte aligned
    b = r.standard_normal((k, n)).astype(np.float32)
    c0 = r.standard_normal((m, n)).astype(np.float32)
    out = gemm(capi, 0, 0, m, n, k, a, b, c0=c0, accumulate=1, lda=k + 1)
    assert_close(out, c0 + a[:, :k].astype(np.float64) @ b.astype(np.float64), 1e-4, "accumulate + odd lda")


def test_tensor_core_gemm_is_deterministic(capi):
    r = rng(6)
    a = r.standard_normal((256, 3136)).astype(np.float32)
    b = r.standard_normal((3136, 128)).astype(np.float32)
    assert np.array_equal(gemm(capi, 0, 0, 256, 128, 3136, a, b), gemm(capi, 0, 0, 256, 128, 3136, a, b))


# ---- operands split into 16-bit parts (k_gemm_parts.cu): work of 2^27 and more, more than one wave of 128 x 64 tiles -------------
# Only the fourth has no short segments at its ends, by which the largest element of a segment tells that the range is wide.
PARTS = [(1300, 1000, 129), (1281, 1089, 257), (2049, 640, 1055), (1024, 1216, 2080), (1409, 901, 300)]
# Error relative to |A| |B|: at most 32 additions to an accumulator between two roundings, each truncated (2^-23), the parts' own 2^-22 and
# the sums over the chunks.
PARTS_BOUND = 32 * 2.0**-23 + 2.0**-21


def parts_error(got, A, B):
    A, B = A.astype(np.float64), B.astype(np.float64)
    return float(np.max(np.abs(got - A @ B) / (np.abs(A) @ np.abs(B))))


@pytest.mark.parametrize("inputs", ["normal", "one row far below the rest", "scales that cancel along the reduction", "tiny times huge", 28, 31, 35, 40, 50])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", PARTS, ids=str)
def test_product_of_parts(capi, m, n, k, ta, tb, inputs):
    r = rng(m + n + k)
    A, B = r.standard_normal((m, k)).astype(np.float32), r.standard_normal((k, n)).astype(np.float32)
    if inputs == "one row far below the rest":
        A[m // 2] *= np.float32(2.0**-40)
    elif inputs == "scales that cancel along the reduction":
        s = np.exp2(np.round(np.linspace(-30, 30, k))).astype(np.float32)
        A, B = A * s, B / s[:, None]
    elif inputs == "tiny times huge":
        A, B = A * np.float32(1e-25), B * np.float32(3e20)
    elif inputs != "normal":  # magnitudes spread over so many powers of two, in every row and column, and columns that give each the same weight
        A = (np.exp2(r.uniform(-inputs / 2, inputs / 2, (m, k))) * r.choice([-1, 1], (m, k))).astype(np.float32)
        B = np.ascontiguousarray((1 / np.abs(A[np.arange(n) % m])).T)
    before = capi.launches()
    got = gemm(capi, ta, tb, m, n, k, np.ascontiguousarray(A.T) if ta else A, np.ascontiguousarray(B.T) if tb else B)
    assert capi.launches() - before <= 4  # a sample, two parts, perhaps three, the product
    assert parts_error(got, A, B) < PARTS_BOUND


def test_product_of_parts_keeps_infinities_and_nan_apart(capi):
    r = rng(9)
    A, B = r.standard_normal((1300, 300)).astype(np.float32), r.standard_normal((300, 1000)).astype(np.float32)
    B[11] = 1.0  # one 16-bit part: the others are zero and must not meet the infinity
    ref = A.astype(np.float64) @ B
    A[5, 11], A[70, 11], A[1200, 3] = np.inf, -np.inf, np.nan
    got = gemm(capi, 0, 0, 1300, 1000, 300, A, B)
    assert np.all(got[5] == np.inf) and np.all(got[70] == -np.inf) and np.all(np.isnan(got[1200]))
    rest = np.delete(np.arange(1300), [5, 70, 1200])
    assert_close(got[rest], ref[rest], 1e-4, "rows without them")


def test_product_of_parts_accumulate_bias_activation_and_ragged_rows(capi):
    r = rng(10)
    m, n, k = 1301, 1003, 259
    A, B, c0, bias = (r.standard_normal(s).astype(np.float32) for s in ((m, k + 2), (k, n + 3), (m, n), (n,)))
    ref = A[:, :k].astype(np.float64) @ B[:, :n]
    out = gemm(capi, 0, 0, m, n, k, A, B, c0=c0, accumulate=1, lda=k + 2, ldb=n + 3)
    assert_close(out, c0 + ref, 1e-4, "accumulate")
    dev, dc = [capi.to_device(v) for v in (A, B, bias)], capi.empty((m, n))
    capi.call("gemm_bias_act", C.c_int64(m), C.c_int64(n), C.c_int64(k), dev[0].ptr, C.c_int64(k + 2), dev[1].ptr, C.c_int64(n + 3), dev[2].ptr,
              C.c_int(1), dc.ptr, C.c_int64(n))
    assert_close(dc.numpy(), np.maximum(ref + bias, 0), 1e-4, "bias and relu")


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("m,k,n", [(1300, 1101, 1203), (1153, 1280, 1536)])
def test_both_gradients_of_a_product_of_parts(capi, m, k, n, accumulate):
    r = rng(m + n)
    a, b, g, db0 = (r.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n), (k, n)))
    dev, da, db = [capi.to_device(v) for v in (a, b, g)], capi.empty((m, k)), capi.to_device(db0)
    capi.call("matmul_backward_accumulate" if accumulate else "matmul_backward", *[d.ptr for d in dev], C.c_int64(m), C.c_int64(k), C.c_int64(n), da.ptr,
              db.ptr)
    assert parts_error(da.numpy(), g, b.T) < PARTS_BOUND
    got = db.numpy().astype(np.float64) - (db0 if accumulate else 0)
    assert parts_error(got, a.T, g) < PARTS_BOUND + (2.0**-22 if accumulate else 0)
