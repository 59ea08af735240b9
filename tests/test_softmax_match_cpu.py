"""Which written-out softmaxes the planner replaces with the row kernel: exactly the chain over the last dimension of an f32
value whose steps nothing else reads.  Everything near it keeps the general kernels (no GPU needed: the launch plan is text)."""
import pytest

import ryft_b200
from ryft_b200.stablehlo import Builder


def program(variant):
    shape, dt, axis = [12, 40], "f32", 1
    if variant == "bf16":
        dt = "bf16"
    if variant == "first dimension":
        axis = 0
    b = Builder()
    x = b.arg(shape, dt)
    y = b.transpose(b.arg([40, 12], dt), [1, 0]) if variant == "transposed operand" else x
    keep = [1 - axis]
    m = b.reduce(y, b.constant(0.0 if variant == "maximum from zero" else float("-inf"), [], dt), "minimum" if variant == "minimum" else "maximum", [axis])
    e = b.exponential(b.subtract(y, b.broadcast_in_dim(m, keep, shape)))
    s = b.reduce(y if variant == "sum of the operand" else e, b.constant(1.0 if variant == "sum from one" else 0.0, [], dt), "add", [axis])
    q = b.divide(e, b.broadcast_in_dim(s, keep, shape))
    outs = [q]
    if variant == "narrowed":
        outs = [b.convert(q, "bf16")]
    if variant == "narrowed, quotient read as well":
        outs = [b.convert(q, "bf16"), b.add(q, q)]
    if variant == "maximum returned":
        outs.append(m)
    if variant == "exponentials returned":
        outs.append(e)
    if variant == "sum read":
        outs.append(b.log(s))
    if variant == "operand read":
        outs.append(b.tanh(y))
    return b.build(*outs)


@pytest.mark.parametrize("variant,taken", [("plain", True), ("narrowed", True), ("narrowed, quotient read as well", True), ("transposed operand", True), ("operand read", True),
                                           ("bf16", False), ("first dimension", False), ("maximum from zero", False), ("minimum", False), ("sum from one", False),
                                           ("sum of the operand", False), ("maximum returned", False), ("exponentials returned", False), ("sum read", False)])
def test_row_softmax_match(variant, taken):
    plan = ryft_b200.plan_dump(program(variant))
    assert ("softmax softmax" in plan) == taken, plan
