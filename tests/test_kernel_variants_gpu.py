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


# pieces of fewer rows than a CTA has thread rows: one row, a power of two, one more, columns with and without vectors, in every
# element kind, with a program in front of the reduction and a consumer behind it
@pytest.mark.parametrize("shape", [(1000, 1, 5), (3000, 8, 3), (77, 9, 24), (300, 16, 16), (5, 33, 136), (1, 2, 2)])
@pytest.mark.parametrize("dtype,body,fused", [("f32", "add", False), ("f32", "add", True), ("bf16", "maximum", False), ("i32", "add", False), ("f32", "minimum", True)])
def test_column_reduction_of_few_rows(client, shape, dtype, body, fused):
    b = Builder()
    x = b.arg(shape, dtype)
    init = b.constant({"add": 0 if dtype == "i32" else 0.0, "maximum": float("-inf"), "minimum": float("inf")}[body], [], dtype)
    r = b.reduce(b.multiply(x, x) if fused else x, init, body, [1])
    text = b.build(b.convert(b.multiply(r, b.splat(0.5, r)), "bf16") if fused else r)
    g = np.random.default_rng(8)
    v = g.integers(-1000, 1000, size=shape).astype(np.int32) if dtype == "i32" else g.standard_normal(shape, dtype=np.float32).astype(configs.np_dtype(dtype))
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


# the row sums are no less exact than those of the two reductions and two elementwise passes that the kernel stands for, in each
# of its width classes (the maximum, the exponentials and the quotients are the same values)
@pytest.mark.parametrize("n", [512, 1024, 2048, 4096, 8192, 16384])
def test_row_softmax_is_as_exact_as_the_chain(client, monkeypatch, n):
    from helpers import run_gpu
    rows = 1 << 23 >> (n.bit_length() - 1)
    x = np.random.default_rng(13).standard_normal((rows, n), dtype=np.float32) * np.float32(3)
    e = np.exp(x.astype(np.float64) - x.max(axis=1, keepdims=True))
    want = e / e.sum(axis=1, keepdims=True)
    error = {}
    for fused in ("1", "0"):
        monkeypatch.setenv("B2X_FUSED_SOFTMAX", fused)
        (got,) = run_gpu(client, softmax_program((rows, n)), [x])
        error[fused] = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert error["1"] <= error["0"], error


def test_row_softmax_of_a_value_that_is_also_returned(client):
    shape = (6, 200)
    check_program(client, softmax_program(shape, extra=True), [np.random.default_rng(4).standard_normal(shape, dtype=np.float32)], "softmax, operand returned", f32_tol=1e-6)


# CUDA-core products: one tile, K cut over 2, 4 and 8 CTAs, 64- and 128-row tiles with ragged edges, all four operand forms
@pytest.mark.parametrize("B,M,K,N", [(1, 2, 3, 2), (1, 1, 2049, 1), (1, 65, 127, 63), (1, 8, 2048, 9), (1, 130, 300, 129), (1, 700, 131, 701), (1, 1290, 129, 1283), (3, 70, 515, 33),
                                     (1030, 3, 5, 7)])
@pytest.mark.parametrize("dtype,lc,rc", [("f32", 1, 0), ("bf16", 0, 1), ("f16", 1, 1), ("f32", 0, 0), ("i32", 1, 0), ("i8", 0, 1)])
def test_cuda_core_product(client, B, M, K, N, dtype, lc, rc):
    import ryft_b200
    ls, rs = ([B, M, K] if lc else [B, K, M]), ([B, N, K] if rc else [B, K, N])
    b = Builder()
    x = b.arg(ls, dtype); y = b.arg(rs, dtype)
    text = b.build(b.dot_general(x, y, ([0], [0]), ([2 if lc else 1], [2 if rc else 1]), out_dtype="f32" if dtype in ("f32", "bf16", "f16") else "i32"))
    assert " simt" in ryft_b200.plan_dump(text)
    r = np.random.default_rng(9)
    npdt = configs.np_dtype(dtype)
    ins = [r.integers(-100, 100, size=s).astype(npdt) if dtype[0] == "i" else r.standard_normal(s, dtype=np.float32).astype(npdt) for s in (ls, rs)]
    # products of 16-bit values are exact in f32 and an f32 product rounds with 2^-24; K <= 2049 sums do so as well, with random signs
    check_program(client, text, ins, f"{dtype} {B}x{M}x{K}x{N}", f32_tol=1e-6)


# the same kernel's fused epilogues, four columns and one column per run of the program
@pytest.mark.parametrize("M,K,N", [(100, 520, 136), (77, 640, 61), (1501, 40, 1203)])
def test_cuda_core_product_with_epilogue(client, M, K, N):
    import ryft_b200
    b = Builder()
    x = b.arg([M, K], "bf16"); y = b.arg([K, N], "bf16"); bias = b.arg([N], "f32")
    d = b.dot_general(x, y, ([], []), ([1], [0]), out_dtype="f32")
    s = b.add(d, b.broadcast_in_dim(bias, [1], [M, N]))
    text = b.build(b.tanh(s), b.convert(s, "bf16"))
    assert " simt" in ryft_b200.plan_dump(text)
    r = np.random.default_rng(10)
    ins = [(r.standard_normal(s, dtype=np.float32) * np.float32(0.2)).astype(BF16) for s in ((M, K), (K, N))] + [r.standard_normal((N,), dtype=np.float32)]
    check_program(client, text, ins, f"epilogue {M}x{K}x{N}", f32_tol=1e-6)


# which of the two attention kernels takes a problem: they round the weights against different maxima, so their results tell
# them apart.  Up to one tile per SM (148) and one above, causal up to two per SM and one above, unmasked long 128-wide heads
@pytest.mark.parametrize("B,H,S,D,causal,form", [(1, 74, 200, 64, False, "tile"), (1, 75, 200, 64, False, "persistent"), (2, 12, 1000, 64, False, "persistent"),
                                                 (1, 148, 200, 64, False, "persistent"), (1, 148, 200, 64, True, "tile"), (1, 149, 200, 64, True, "persistent"),
                                                 (1, 19, 1000, 128, False, "persistent"), (1, 19, 1930, 128, False, "tile"), (1, 40, 1930, 64, False, "persistent")])
def test_attention_form(client, monkeypatch, B, H, S, D, causal, form):
    from helpers import run_gpu
    text, ins = configs.c3_program(B, H, S, D, causal=causal), configs.c3_inputs(B, H, S, D)
    monkeypatch.delenv("B2X_ATTENTION_KERNEL", raising=False)
    (chosen,) = run_gpu(client, text, ins)
    got = {}
    for f in ("tile", "persistent"):
        monkeypatch.setenv("B2X_ATTENTION_KERNEL", f)
        (got[f],) = run_gpu(client, text, ins)
    assert not np.array_equal(got["tile"].view(np.int16), got["persistent"].view(np.int16))
    assert np.array_equal(chosen.view(np.int16), got[form].view(np.int16))


# the order in which query tiles are dealt out within one group of heads, both kernel forms on either side of the rule between
# them; rows and heads that are missed or computed twice show as wrong rows
@pytest.mark.parametrize("B,H,S,D,causal", [(1, 5, 300, 64, True), (1, 37, 1100, 64, True), (1, 19, 2100, 128, True), (2, 10, 2050, 128, False)])
def test_attention_tile_order(client, B, H, S, D, causal):
    from helpers import run_gpu
    q, k, v = configs.c3_inputs(B, H, S, D)
    (got,) = run_gpu(client, configs.c3_program(B, H, S, D, causal=causal), [q, k, v])
    got = got.astype(np.float32).reshape(B * H, S, D)
    q, k, v = (t.astype(np.float32).reshape(B * H, S, D) for t in (q, k, v))
    for h in range(B * H):
        s = (q[h] @ k[h].T) * np.float32(1.0 / np.sqrt(D))
        if causal:
            s[np.triu_indices(S, 1)] = -np.inf
        e = np.exp(s - s.max(axis=1, keepdims=True))
        p = e / e.sum(axis=1, keepdims=True)
        want = p @ v[h]
        # the weights and the result are rounded to bf16 once each: 2^-9 of sum p |v| and of the result, times two for ties
        bound = 2 ** -8 * (p @ np.abs(v[h])) + 2 ** -7 * np.abs(want) + 1e-6
        assert (np.abs(got[h] - want) <= bound).all(), (h, float(np.abs(got[h] - want).max()))


# f32 products on the tensor cores: both halves of a k-block in one stage, K that ends inside a block, operands contiguous along
# either dimension, batches, all three tile widths
@pytest.mark.parametrize("B,M,K,N,lc,rc", [(1, 128, 32, 64, 1, 0), (1, 200, 100, 264, 1, 1), (3, 136, 44, 72, 0, 0), (2, 264, 132, 136, 0, 1), (1, 1500, 260, 1032, 1, 0),
                                           (1, 2176, 72, 2056, 0, 0)])
def test_f32_product_on_tensor_cores(client, B, M, K, N, lc, rc):
    import ryft_b200
    ls, rs = ([B, M, K] if lc else [B, K, M]), ([B, N, K] if rc else [B, K, N])
    b = Builder()
    x = b.arg(ls, "f32"); y = b.arg(rs, "f32")
    text = b.build(b.dot_general(x, y, ([0], [0]), ([2 if lc else 1], [2 if rc else 1])))
    assert "3xtf32" in ryft_b200.plan_dump(text)
    r = np.random.default_rng(12)
    ins = [r.standard_normal(s, dtype=np.float32) for s in (ls, rs)]
    # the tensor cores add with truncation: 1.15e-8 of the result for every k (three chains of eight products per addition),
    # and the halves leave out 2^-22 of a product
    check_program(client, text, ins, f"f32 {B}x{M}x{K}x{N} {lc}{rc}", f32_tol=1e-6 + 1.5e-8 * K)


# infinities and NaN in f32 operands of the tensor-core product: beside values that are exact in 11 bits (whose low half is
# zero), beside zeros, of both signs in one sum, a NaN whose set bits all lie below them, through the bulk-store and the
# interpreted epilogue, with edges of tiles and more than one tile
@pytest.mark.parametrize("B,M,K,N,lc,rc", [(1, 128, 64, 64, 1, 0), (1, 200, 100, 264, 1, 1), (2, 136, 40, 136, 0, 0), (1, 1500, 260, 1032, 0, 1)])
@pytest.mark.parametrize("epilogue", [False, True])
def test_f32_product_of_non_finite_values(client, B, M, K, N, lc, rc, epilogue):
    import ryft_b200
    ls, rs = ([B, M, K] if lc else [B, K, M]), ([B, N, K] if rc else [B, K, N])
    b = Builder()
    x = b.arg(ls, "f32"); y = b.arg(rs, "f32")
    d = b.dot_general(x, y, ([0], [0]), ([2 if lc else 1], [2 if rc else 1]))
    text = b.build(b.multiply(b.maximum(d, b.splat(-2.0, d)), b.splat(0.5, d)) if epilogue else d)
    assert "3xtf32" in ryft_b200.plan_dump(text)
    r = np.random.default_rng(14)
    # half of the values are small whole numbers, zero among them
    a, c = (np.where(r.random(s) < 0.5, r.integers(-2, 3, size=s), r.standard_normal(s)).astype(np.float32) for s in ([B, M, K], [B, K, N]))
    inf = np.float32(np.inf)
    a[0, 3, 5] = inf                              # one infinity: its row is infinite, or NaN where it meets a zero
    a[-1, M - 1, K - 1] = -inf
    a[0, 40, 1] = inf; a[0, 40, K // 2] = -inf    # two in one row: the signs of the other operand decide
    c[0, 7, 9] = -inf
    c[-1, 0, N - 1] = inf
    c[0, 5, 20] = inf                             # meets the infinity of row 3
    a[0, 70, 2] = np.array([0x7f800001], np.uint32).view(np.float32)[0]
    c[-1, 3, 33] = np.nan
    ins = [a if lc else np.ascontiguousarray(a.swapaxes(1, 2)), np.ascontiguousarray(c.swapaxes(1, 2)) if rc else c]
    with np.errstate(invalid="ignore"):
        got = check_program(client, text, ins, f"f32 {B}x{M}x{K}x{N} {lc}{rc}", f32_tol=1e-6 + 1.5e-8 * K)
    assert np.isinf(got[0]).sum() > 100


# clustered column reductions: a 16-bit sum over several CTAs, and a consumer that the first CTA of the cluster runs; either side
# of the rule between one launch and two
@pytest.mark.parametrize("R,N", [(8192, 520), (4100, 2568), (8192, 2304), (8192, 2312)])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("consumer", [False, True])
def test_clustered_column_sum(client, R, N, dtype, consumer):
    b = Builder()
    x = b.arg([R, N], dtype)
    r = b.reduce(b.convert(x, "f32") if dtype != "f32" else x, b.constant(0.0, [], "f32"), "add", [0])
    text = b.build(b.convert(b.multiply(r, b.splat(0.5, r)), "bf16") if consumer else r)
    v = np.random.default_rng(18).standard_normal((R, N), dtype=np.float32).astype(configs.np_dtype(dtype))
    check_program(client, text, [v], f"column sum {dtype} {R}x{N}", f32_tol=1e-6)


# several groups of heads (as many to a group as have 32 MiB of keys and values): a shorter last group, one head per group, and
# one group as the limit, in both kernel forms, with every row of every head checked
@pytest.mark.parametrize("BH,Sq,Sk,D,per_group", [(5, 300, 20000, 128, 3), (3, 200, 40000, 128, 1), (7, 257, 40000, 64, 3), (2, 300, 32768, 128, 2)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("form", ["tile", "persistent"])
def test_attention_groups_of_heads(monkeypatch, BH, Sq, Sk, D, per_group, causal, form):
    import ctypes as C

    import torch

    from ryft_b200 import kernels

    class Args(C.Structure):
        _fields_ = [("q", C.c_void_p), ("k", C.c_void_p), ("v", C.c_void_p), ("o", C.c_void_p), ("BH", C.c_int64), ("Sq", C.c_int64), ("Sk", C.c_int64), ("D", C.c_int64),
                    ("scale", C.c_float), ("causal", C.c_int)]

    assert max(1, min(BH, (32 << 20) // (Sk * D * 4))) == per_group
    lib = kernels.load()
    monkeypatch.setenv("B2X_ATTENTION_KERNEL", form)
    g = torch.Generator(device="cuda").manual_seed(11)
    q, k, v = (torch.randn((BH, n, D), generator=g, device="cuda").bfloat16() for n in (Sq, Sk, Sk))
    o = torch.full((BH, Sq, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = Args(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), BH, Sq, Sk, D, D ** -0.5, int(causal))
    lib.b2x_launch_attention.argtypes = [C.POINTER(Args), C.c_void_p, C.c_void_p]
    assert lib.b2x_launch_attention(C.byref(a), status.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert status.item() == 0
    for h in range(BH):
        s = (q[h].double() @ k[h].double().T) * D ** -0.5
        if causal:
            s.masked_fill_(torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        w = torch.softmax(s, dim=1)
        want = w @ v[h].double()
        # one rounding of the weights and one of the result to bf16, as above; the row sums are exact to 2^-20 or so
        bound = 2 ** -8 * (w @ v[h].double().abs()) + 2 ** -7 * want.abs() + 1e-6
        assert ((o[h].double() - want).abs() <= bound).all(), (h, (o[h].double() - want).abs().max().item())


# the threefold split of f32 operands for a single product over 3 K: [hi | hi | lo] and [hi | lo | hi], bit for bit
@pytest.mark.parametrize("B,M,N,K,lc,rc", [(1, 3, 5, 7, 1, 0), (2, 33, 130, 128, 0, 1), (1, 70, 129, 300, 1, 1), (3, 128, 32, 33, 0, 0)])
def test_threefold_split(B, M, N, K, lc, rc):
    import ctypes as C

    import torch

    from ryft_b200 import kernels

    class Args(C.Structure):
        _fields_ = [("a", C.c_void_p), ("b", C.c_void_p), ("elem", C.c_uint8)] + [(n, C.c_int64) for n in (
            "batch", "M", "N", "K", "a_batch_stride", "a_row_stride", "a_k_stride", "b_batch_stride", "b_row_stride", "b_k_stride")]

    lib = kernels.load()
    r = np.random.default_rng(15)
    a, b = r.standard_normal((B, M, K), dtype=np.float32), r.standard_normal((B, N, K), dtype=np.float32)
    da, db = (torch.from_numpy(np.ascontiguousarray(x if c else x.swapaxes(1, 2))).cuda() for x, c in ((a, lc), (b, rc)))
    sa, sb = (torch.full((B, rows, 3 * K), float("nan"), device="cuda") for rows in (M, N))
    args = Args(da.data_ptr(), db.data_ptr(), kernels.EL_F32, B, M, N, K, M * K, K if lc else 1, 1 if lc else M, N * K, K if rc else 1, 1 if rc else N)
    lib.b2x_launch_split_f32.argtypes = [C.POINTER(Args), C.c_void_p, C.c_void_p, C.c_void_p]
    assert lib.b2x_launch_split_f32(C.byref(args), sa.data_ptr(), sb.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0

    def cut(x):
        return (x.view(np.uint32) & np.uint32(0xffffe000)).view(np.float32)
    for got, x, order in ((sa, a, (0, 0, 1)), (sb, b, (0, 1, 0))):
        halves = (cut(x), cut(x - cut(x)))
        assert np.array_equal(got.cpu().numpy(), np.concatenate([halves[i] for i in order], axis=2))


# a row softmax between other kernels: its operand made by a product and an elementwise step, or by a reduction; its result read
# by a product
@pytest.mark.parametrize("B,S,D", [(3, 70, 40), (2, 136, 64)])
def test_row_softmax_between_products(client, B, S, D):
    import ryft_b200
    b = Builder()
    x = b.arg([B, S, D], "f32"); y = b.arg([B, S, D], "f32")
    s = b.dot_general(x, y, ([0], [0]), ([2], [2]))
    s = b.multiply(s, b.splat(0.125, s))
    m = b.reduce(s, b.constant(float("-inf"), [], "f32"), "maximum", [2])
    e = b.exponential(b.subtract(s, b.broadcast_in_dim(m, [0, 1], [B, S, S])))
    l = b.reduce(e, b.constant(0.0, [], "f32"), "add", [2])
    q = b.divide(e, b.broadcast_in_dim(l, [0, 1], [B, S, S]))
    text = b.build(b.dot_general(q, y, ([0], [0]), ([2], [1])))
    assert "softmax softmax" in ryft_b200.plan_dump(text)
    r = np.random.default_rng(16)
    # a difference of 1e-6 in the scores (f32 sums over D) is one of 1e-6 in the weights
    check_program(client, text, [r.standard_normal((B, S, D), dtype=np.float32) for _ in range(2)], f"attention in f32 {B}x{S}x{D}", f32_tol=5e-6)


def test_row_softmax_of_a_reduction(client):
    import ryft_b200
    shape = [37, 50, 130]
    b = Builder()
    x = b.arg(shape, "f32")
    y = b.reduce(x, b.constant(0.0, [], "f32"), "add", [1])
    m = b.reduce(y, b.constant(float("-inf"), [], "f32"), "maximum", [1])
    e = b.exponential(b.subtract(y, b.broadcast_in_dim(m, [0], [37, 130])))
    s = b.reduce(e, b.constant(0.0, [], "f32"), "add", [1])
    text = b.build(b.divide(e, b.broadcast_in_dim(s, [0], [37, 130])))
    assert "softmax softmax" in ryft_b200.plan_dump(text)
    # the sums of 50 normals (up to 30) round with 2^-24 of themselves a few times: as much in the exponentials
    check_program(client, text, [np.random.default_rng(17).standard_normal(shape, dtype=np.float32)], "softmax of a reduction", f32_tol=1e-5)


# kernels that start early reuse the blocks of one arena, execution after execution and on other arguments each time: what one
# reads is what the kernels in front of it have written
def test_back_to_back_executions_reuse_one_arena(client):
    from ryft_b200 import pjrt
    n = 160
    b = Builder()
    x = b.arg([n, n], "f32"); w = b.arg([n, n], "bf16")
    y = x
    for _ in range(4):
        h = b.dot_general(b.convert(y, "bf16"), w, ([], []), ([1], [0]), out_dtype="f32")
        t = b.reduce(b.multiply(h, h), b.constant(0.0, [], "f32"), "add", [0])
        y = b.tanh(b.subtract(h, b.broadcast_in_dim(b.multiply(t, b.splat(1.0 / n, t)), [1], [n, n])))
    exe = client.compile(pjrt.Program.mlir(b.build(y)))
    r = np.random.default_rng(19)
    wb = client.buffer((r.standard_normal((n, n), dtype=np.float32) * np.float32(n ** -0.5)).astype(BF16))
    xs = [client.buffer(r.standard_normal((n, n), dtype=np.float32)) for _ in range(3)]
    alone = []
    for xb in xs:
        out = exe.execute([pjrt.ExecutionDeviceInputs([xb, wb])])[0]
        out.done.await_()
        alone.append(out.outputs[0].to_numpy())
    queued = [exe.execute([pjrt.ExecutionDeviceInputs([xs[i % 3], wb])])[0] for i in range(60)]
    for i, out in enumerate(queued):
        assert np.array_equal(out.outputs[0].to_numpy(), alone[i % 3]), i


# two executables on two threads read one view; the view goes away while they are still queued
def test_view_outlives_the_executions_of_two_threads(client):
    import threading

    import torch

    from ryft_b200 import pjrt

    def program(factor):
        b = Builder()
        x = b.arg([1 << 20], "f32")
        y = x
        for _ in range(20):
            y = b.add(b.multiply(y, b.splat(0.5, y)), b.splat(factor, y))
        return b.build(y)
    exes = [client.compile(pjrt.Program.mlir(program(f))) for f in (0.25, 0.75)]
    for _ in range(10):
        t = torch.ones(1 << 20, device="cuda")
        torch.cuda.synchronize()
        view = client.view_of_device_buffer(t.data_ptr(), pjrt.BufferType.F32, [1 << 20], keep=t)
        results = [[], []]

        def work(i):
            for _ in range(20):
                results[i].append(exes[i].execute([pjrt.ExecutionDeviceInputs([view])])[0])
        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        del view                                  # waits for every reader
        t.fill_(float("nan"))
        torch.cuda.synchronize()
        for i, f in enumerate((0.25, 0.75)):
            want = np.float32(1.0)
            for _ in range(20):
                want = np.float32(want * np.float32(0.5)) + np.float32(f)
            for out in results[i]:
                assert (out.outputs[0].to_numpy() == want).all()
