"""The heads' norm with a head's values held in registers (csrc/recurrent.cu): its lanes per head, its remainders and the way back to
one value at a time."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _ref(raw, dv, eps, m, weight, gate, act):
    x = raw.double()[..., :dv]
    if m is not None:
        x = x / (torch.maximum(raw.double()[..., dv].abs(), m.double()) + 1e-6)[..., None]
    x = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)).flatten(1)
    if weight is not None:
        x = x * weight.double()
    if act:
        x = x * torch.sigmoid(gate.double()) * (1 if act == "sigmoid" else gate.double())
    return x


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,H,dv,extra,shift,act,weighted", [
    (1, 1, 4, 0, 0, "silu", True), (3, 5, 32, 0, 0, None, False), (5, 3, 36, 0, 0, "sigmoid", True), (2, 7, 64, 0, 0, "silu", True),
    (3, 3, 100, 0, 0, "silu", False), (3, 1, 128, 0, 0, "sigmoid", True), (2, 3, 132, 0, 0, "silu", True), (3, 2, 256, 0, 0, None, True),
    (2, 3, 260, 0, 0, "silu", True), (3, 3, 30, 0, 0, "silu", True), (3, 3, 64, 0, 3, "silu", True), (5, 3, 64, 1, 0, "sigmoid", True),
    (3, 3, 128, 1, 0, "silu", True), (1, 5, 129, 1, 0, None, True), (3, 3, 256, 1, 0, "silu", True), (2, 2, 300, 1, 0, "silu", True)])
def test_a_head_held_in_registers(dtype, rows, H, dv, extra, shift, act, weighted):
    """extra: a denominator behind the values (rows of raw then start anywhere); shift: a gate off a vector's boundary."""
    from longbow_quarrel_b200.kernels import ops
    g = torch.Generator().manual_seed(dv + rows)
    raw = 3.0 * torch.randn(rows, H, dv + extra, generator=g)
    m = torch.rand(rows, H, generator=g) if extra else None
    weight = 1 + 0.3 * torch.randn(H * dv, generator=g) if weighted else None
    gate = torch.randn(rows, H * dv + 8, generator=g).to(dtype)
    on = lambda t: None if t is None else t.to(DEV)
    got = ops.head_norm_gate(on(raw), dv, 1e-5, dtype, exp_neg_m=on(m), weight=on(weight),
                             gate=on(gate)[:, shift:shift + H * dv] if act else None, act=act)
    want = _ref(raw, dv, 1e-5, m, weight, gate[:, shift:shift + H * dv], act)
    # the sum of squares: at most 10 additions in a chain and 5 across lanes; ten more roundings, expf within 2 units; bfloat16: half a unit
    assert bool(((got.cpu().double() - want).abs() <= want.abs() * (32 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) + 1e-30).all())
    ops.check_status()
