"""The work that a program of this framework hands to the plugin, as cases that can be timed and compared.

Every case is one StableHLO program, compiled through `Client.compile` and run through `LoadedExecutable.execute` on
arguments that are resident on the GPU, the way a training or serving loop keeps them: a contraction in each element
type, a dense layer with its bias and activation, attention, a whole training step, and the elementwise and reduce
programs that run between them.  The results come back as torch tensors over the plugin's own output buffers.
"""
from __future__ import annotations

import functools
import math

import torch

from ryft_b200 import configs, pjrt
from ryft_b200.stablehlo import Builder

_TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_TYPE = {"f32": pjrt.BufferType.F32, "bf16": pjrt.BufferType.BF16, "f16": pjrt.BufferType.F16}
_SIZE = {"f32": 4, "bf16": 2, "f16": 2}


# ---- the cases ---------------------------------------------------------------------------------------------------------

def listed():
    return [
        # a contraction of a few elements, as in the dimension-number tests: nothing but the cost of a call
        {"name": "dot_tiny", "kind": "dot", "M": 17, "K": 33, "N": 5, "dtype": "f32", "lc": 1, "rc": 0},
        # the f32 matrix product of the first benchmark configuration: a small layer in the default element type
        {"name": "dot_f32", "kind": "dot", "M": 512, "K": 768, "N": 512, "dtype": "f32", "lc": 1, "rc": 0},
        # an f32 weight gradient (both operands contracted over their first dimension) at the width of the large MLP
        {"name": "dot_f32_large", "kind": "dot", "M": 4096, "K": 2048, "N": 4096, "dtype": "f32", "lc": 0, "rc": 0},
        # a 16-bit contraction whose sizes are multiples of nothing, as vocabularies and sequence lengths often are
        {"name": "dot_bf16_odd", "kind": "dot", "M": 1023, "K": 777, "N": 1001, "dtype": "bf16", "lc": 1, "rc": 0},
        # batched dense layer with bias and activation, the second benchmark configuration
        {"name": "dense_tanh", "kind": "dense", "B": 32, "M": 2048, "K": 128, "N": 2048},
        # causal attention over long sequences (training, prefill), the third benchmark configuration
        {"name": "attention_causal", "kind": "attention", "B": 4, "H": 32, "S": 4096, "D": 128, "causal": True},
        # attention without a mask over a sequence that ends inside a tile (an encoder), with the narrower head
        {"name": "attention_full", "kind": "attention", "B": 2, "H": 12, "S": 1000, "D": 64, "causal": False},
        # a training step of a small model with ragged sizes: every launch counts
        {"name": "mlp_small", "kind": "mlp", "T": 200, "D": 136, "F": 264},
        # the training step of the headline benchmark: forward, backward, loss
        {"name": "mlp_large", "kind": "mlp", "T": 8192, "D": 4096, "F": 16384},
        # bias and activation as a program of its own, at the size of the dense layer above
        {"name": "bias_tanh", "kind": "bias_tanh", "B": 32, "M": 2048, "N": 2048},
        # the gradient of a bias (column sums) at the size of the training step's output
        {"name": "bias_gradient", "kind": "column_sum", "T": 8192, "D": 4096},
        # softmax written out over rows (two reductions and the elementwise work between them)
        {"name": "softmax", "kind": "softmax", "R": 8192, "N": 4096},
    ]


def _size(rng, low, high, multiple=1):
    """A size whose logarithm is spread evenly over [low, high], rounded to `multiple`."""
    n = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(low, min(high, int(round(n / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(["dot", "dot", "dense", "attention", "mlp", "bias_tanh", "column_sum", "softmax"])
    # half of the sizes are multiples of eight, the others are whatever they happen to be
    m = rng.choice([1, 8])
    if kind == "dot":
        top = 2048 if m == 1 else 4096
        return {"kind": kind, "M": _size(rng, 8, top, m), "K": _size(rng, 8, 2048, m), "N": _size(rng, 8, top, m),
                "dtype": rng.choice(["f32", "bf16", "f16"]), "lc": rng.choice([0, 1]), "rc": rng.choice([0, 1])}
    if kind == "dense":
        return {"kind": kind, "B": _size(rng, 1, 32), "M": _size(rng, 64, 2048, m), "K": _size(rng, 64, 1024, 8), "N": _size(rng, 64, 2048, 8)}
    if kind == "attention":
        return {"kind": kind, "B": _size(rng, 1, 4), "H": _size(rng, 1, 32), "S": _size(rng, 64, 4096, m), "D": rng.choice([64, 128]),
                "causal": rng.choice([True, False])}
    if kind == "mlp":
        return {"kind": kind, "T": _size(rng, 64, 8192, m), "D": _size(rng, 64, 2048, 8), "F": _size(rng, 128, 8192, 8)}
    if kind == "bias_tanh":
        return {"kind": kind, "B": _size(rng, 1, 32), "M": _size(rng, 8, 2048), "N": _size(rng, 8, 2048, m)}
    if kind == "column_sum":
        return {"kind": kind, "T": _size(rng, 8, 8192), "D": _size(rng, 8, 4096, m)}
    return {"kind": kind, "R": _size(rng, 8, 8192), "N": _size(rng, 16, 4096, m)}


# ---- programs ------------------------------------------------------------------------------------------------------------

def _softmax_program(R, N):
    b = Builder()
    x = b.arg([R, N], "f32")
    m = b.reduce(x, b.constant(float("-inf"), [], "f32"), "maximum", [1])
    e = b.exponential(b.subtract(x, b.broadcast_in_dim(m, [0], [R, N])))
    s = b.reduce(e, b.constant(0.0, [], "f32"), "add", [1])
    return b.build(b.divide(e, b.broadcast_in_dim(s, [0], [R, N])))


def _column_sum_program(T, D):
    b = Builder()
    x = b.arg([T, D], "f32")
    return b.build(b.reduce(x, b.constant(0.0, [], "f32"), "add", [0]))


def _dot_program(M, K, N, dtype, lc, rc):
    b = Builder()
    x = b.arg([M, K] if lc == 1 else [K, M], dtype)
    y = b.arg([K, N] if rc == 0 else [N, K], dtype)
    return b.build(b.dot_general(x, y, ([], []), ([lc], [rc]), out_dtype="f32"))


def _describe(c):
    """(program text, [(argument shape, element type, scale)], [(result shape, element type)]) of a case."""
    k = c["kind"]
    if k == "dot":
        M, K, N, dt = c["M"], c["K"], c["N"], c["dtype"]
        # 16-bit operands carry the scale that keeps results of order one, as activations and weights do
        scale = 1.0 if dt == "f32" else K ** -0.25
        return (_dot_program(M, K, N, dt, c["lc"], c["rc"]),
                [([M, K] if c["lc"] == 1 else [K, M], dt, scale), ([K, N] if c["rc"] == 0 else [N, K], dt, scale)], [([M, N], "f32")])
    if k == "dense":
        B, M, K, N = c["B"], c["M"], c["K"], c["N"]
        return (configs.c2_program(B, M, K, N), [([B, M, K], "bf16", K ** -0.5), ([B, K, N], "bf16", K ** -0.5), ([N], "f32", 0.1)],
                [([B, M, N], "bf16")])
    if k == "attention":
        s = [c["B"], c["H"], c["S"], c["D"]]
        return configs.c3_program(*s, causal=c["causal"]), [(s, "bf16", 1.0)] * 3, [(s, "bf16")]
    if k == "mlp":
        T, D, F = c["T"], c["D"], c["F"]
        return (configs.c4_program(T, D, F), [([T, D], "bf16", 1.0), ([D, F], "bf16", 0.02), ([F, D], "bf16", 0.02)],
                [([D, F], "f32"), ([F, D], "f32"), ([], "f32")])
    if k == "bias_tanh":
        s = [c["B"], c["M"], c["N"]]
        return configs.ew_program(*s), [(s, "f32", 0.1), ([c["N"]], "f32", 0.1)], [(s, "bf16")]
    if k == "column_sum":
        return _column_sum_program(c["T"], c["D"]), [([c["T"], c["D"]], "f32", 1.0)], [([c["D"]], "f32")]
    return _softmax_program(c["R"], c["N"]), [([c["R"], c["N"]], "f32", 3.0)], [([c["R"], c["N"]], "f32")]


# ---- preparing and running -------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _client():
    return pjrt.load_cuda_13_plugin().client({"visible_devices": [0]})


@functools.lru_cache(maxsize=4)
def _executable(text):
    """A program is compiled once, when it is first met, and kept for its later inputs."""
    return _client().compile(pjrt.Program.mlir(text))


class _Result:
    """An output buffer as torch sees it: the memory stays the plugin's and lives as long as the tensor over it."""

    def __init__(self, buffer, shape, dtype):
        self.buffer = buffer
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4" if dtype == "f32" else "<i2", "data": (buffer.device_pointer(), False), "version": 2}


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [(torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(_TORCH[dt]) for shape, dt, scale in _describe(case)[1]]


def prepare(case, seed):
    text, args, results = _describe(case)
    executable = _executable(text)
    tensors = _inputs(case, seed)
    torch.cuda.current_stream().synchronize()
    buffers = [_client().view_of_device_buffer(t.data_ptr(), _TYPE[dt], shape, keep=t) for t, (shape, dt, _) in zip(tensors, args)]
    return {"executable": executable, "arguments": [pjrt.ExecutionDeviceInputs(buffers)], "results": [(tuple(s), dt) for s, dt in results]}


def run(state):
    outputs = state["executable"].execute(state["arguments"])[0].outputs
    stream = torch.cuda.current_stream().cuda_stream
    tensors = []
    for buffer, (shape, dtype) in zip(outputs, state["results"]):
        buffer.wait_until_ready_on_stream(stream)     # what torch does with the tensor comes after the program
        t = torch.as_tensor(_Result(buffer, shape, dtype), device="cuda")
        tensors.append(t if dtype == "f32" else t.view(_TORCH[dtype]))
    return tensors


# ---- what a pass cannot do without, and what it has to yield ----------------------------------------------------------------

def work(case):
    _, args, results = _describe(case)
    size = sum(math.prod(s) * _SIZE[dt] for s, dt, *_ in args + results)
    k = case["kind"]
    if k == "dot":
        flops = 2.0 * case["M"] * case["K"] * case["N"]
    elif k == "dense":
        flops = 2.0 * case["B"] * case["M"] * case["K"] * case["N"]
    elif k == "attention":
        s = case["S"]
        flops = 4.0 * case["B"] * case["H"] * case["D"] * (s * (s + 1) / 2 if case["causal"] else s * s)
    elif k == "mlp":
        flops = 10.0 * case["T"] * case["D"] * case["F"]
    else:
        flops = 0.0
    return {"bytes": float(size), "flops": flops}


def tolerance(case):
    k = case["kind"]
    if k == "dot":
        # f32 operands: three TF32 products of split operands, accumulated by the tensor cores; 16-bit operands are exact
        # products, so only the order (and truncation) of the f32 sums shows
        return {"rel": 5e-5, "max": 1e-3}
    if k in ("dense", "bias_tanh"):
        # one bf16 rounding of the result, and an approximate tanh (2^-11) in front of it
        return {"rel": 5e-3, "max": 2e-2}
    if k == "attention":
        # the softmax weights and the result are rounded to bf16; the first rows of a head are single values, far above the
        # root mean square of the others
        return {"rel": 1e-2, "max": 0.3}
    if k == "mlp":
        # four bf16 roundings follow one another: two evaluations with different orders of summation are 1e-3 apart on dW1
        return {"rel": 5e-3, "max": 1e-1}
    return {"rel": 1e-5, "max": 1e-4}


def _gelu(h):
    """(gelu(h), its derivative) with the tanh form."""
    c0 = math.sqrt(2.0 / math.pi)
    t = torch.tanh(c0 * (h + 0.044715 * h ** 3))
    return 0.5 * h * (1 + t), 0.5 * (1 + t) + 0.5 * h * (1 - t * t) * c0 * (1 + 3 * 0.044715 * h * h)


def exact(case, seed):
    a = _inputs(case, seed)
    k = case["kind"]
    wide = [t.double() for t in a] if k != "attention" else a
    if k == "dot":
        x, y = wide
        return [(x if case["lc"] == 1 else x.T) @ (y if case["rc"] == 0 else y.T)]
    if k == "dense":
        out = torch.empty(case["B"], case["M"], case["N"], dtype=torch.float64, device="cuda")
        for i in range(case["B"]):
            out[i] = torch.tanh(wide[0][i] @ wide[1][i] + wide[2])
        return [out]
    if k == "attention":
        q, key, v = a
        s = case["S"]
        out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
        above = torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1) if case["causal"] else None
        for i in range(case["B"]):
            for j in range(case["H"]):
                p = (q[i, j].double() @ key[i, j].double().T) * (1.0 / math.sqrt(case["D"]))
                if above is not None:
                    p.masked_fill_(above, float("-inf"))
                out[i, j] = torch.softmax(p, dim=1) @ v[i, j].double()
        return [out]
    if k == "mlp":
        # the values that the program converts to bf16 are rounded here as well
        x, w1, w2 = wide
        half = lambda t: t.bfloat16().double()  # noqa: E731
        n = float(case["T"]) * float(case["D"])
        hf = x @ w1
        h, act = half(hf), half(_gelu(hf)[0])
        y = act @ w2
        dy = half(y * (2.0 / n))
        dh = half((dy @ w2.T) * _gelu(h)[1])
        return [x.T @ dh, act.T @ dy, (y * y).sum() / n]
    if k == "bias_tanh":
        return [torch.tanh(wide[0] + wide[1])]
    if k == "column_sum":
        return [wide[0].sum(dim=0)]
    return [torch.softmax(wide[0], dim=1)]
