"""Kernel variants at the sizes where their tiling can go wrong, against the CPU oracle through the PJRT C ABI."""
import numpy as np
import pytest

from ryft_b200 import configs
from ryft_b200.stablehlo import Builder

from helpers import check_program

pytestmark = pytest.mark.gpu
BF16 = configs.BF16


# [A, R, B] reduced over R: one column block and several, ragged ones, fewer rows than thread rows, clusters of every
# size, row splits on top of clusters, columns that allow no vector loads
@pytest.mark.parametrize("shape", [(1, 8192, 4096), (1, 8200, 72), (1, 2048, 33), (1, 5, 4104), (3, 1000, 136), (700, 9, 40), (1, 70000, 8), (2, 4100, 1)])
@pytest.mark.parametrize("dtype,body", [("f32", "add"), ("f32", "maximum"), ("bf16", "maximum"), ("i32", "add"), ("f32", "minimum")])
def test_column_reduction(client, shape, dtype, body):
    if dtype != "f32" and shape[1] * shape[2] > 10_000_000:
        shape = (1, 8192, 520)
    b = Builder()
    x = b.arg(shape, dtype)
    init = b.constant({"add": 0 if dtype == "i32" else 0.0, "maximum": float("-inf"), "minimum": float("inf")}[body], [], dtype)
    text = b.build(b.reduce(x, init, body, [1]))
    r = np.random.default_rng(7)
    v = r.integers(-1000, 1000, size=shape).astype(np.int32) if dtype == "i32" else r.standard_normal(shape, dtype=np.float32).astype(configs.np_dtype(dtype))
    if dtype != "i32" and shape[1] > 7:
        v[0, 7, 0] = np.nan                     # a NaN element makes its column NaN under every body
    # a sum of R normals has size sqrt(R); its partial sums round R / parts times with 2^-24 of at most that size each
    check_program(client, text, [v], f"{body} {dtype} {shape}", f32_tol=1e-6)


def softmax_program(shape, out_dtype="f32", extra=False):
    lead = list(range(len(shape) - 1))
    b = Builder()
    x = b.arg(shape, "f32")
    y = b.multiply(x, b.splat(0.5, x)) if extra else x
    m = b.reduce(y, b.constant(float("-inf"), [], "f32"), "maximum", [len(shape) - 1])
    e = b.exponential(b.subtract(y, b.broadcast_in_dim(m, lead, shape)))
    s = b.reduce(e, b.constant(0.0, [], "f32"), "add", [len(shape) - 1])
    q = b.divide(e, b.broadcast_in_dim(s, lead, shape))
    out = b.convert(q, out_dtype) if out_dtype != "f32" else q
    return b.build(out, y) if extra else b.build(out)


# every width class of the row kernel at its edges, with and without 16-byte rows; one element; the longest row and the
# first one that takes the chain of kernels instead
@pytest.mark.parametrize("shape", [(5, 1), (9, 31), (17, 128), (3, 129), (70, 256), (11, 513), (1024,), (4, 2, 1025), (7, 2048), (3, 4096), (2, 4100), (2, 8193), (1, 16384),
                                   (2, 16385)])
@pytest.mark.parametrize("out_dtype", ["f32", "bf16", "f16"])
def test_row_softmax(client, shape, out_dtype):
    import ryft_b200
    text = softmax_program(shape, out_dtype)
    assert ("softmax softmax" in ryft_b200.plan_dump(text)) == (shape[-1] <= 16384)
    x = np.random.default_rng(3).standard_normal(shape, dtype=np.float32) * np.float32(3)
    if x.ndim == 2 and shape[0] >= 3 and shape[1] > 2:
        x[0, 1] = np.nan
        x[1, :] = -np.inf
        x[2, 2] = -np.inf
    # expf, the f32 sum of up to 16385 positive terms over 256 partial sums and the division: a few units of 2^-24
    check_program(client, text, [x], f"softmax {out_dtype} {shape}", f32_tol=1e-6)


def test_row_softmax_of_a_value_that_is_also_returned(client):
    shape = (6, 200)
    check_program(client, softmax_program(shape, extra=True), [np.random.default_rng(4).standard_normal(shape, dtype=np.float32)], "softmax, operand returned", f32_tol=1e-6)
