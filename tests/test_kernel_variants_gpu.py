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
