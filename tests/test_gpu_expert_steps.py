"""The experts' products of single tokens with several rows of weight at a time (csrc/moe.cu): the same sums as one row at a time."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("gated,block", [(False, 0), (True, 0), (True, 8)])
@pytest.mark.parametrize("T,top,E,D,F", [(1, 2, 3, 8, 8), (1, 6, 7, 256, 264), (3, 6, 9, 264, 1000), (9, 3, 4, 1288, 40), (40, 2, 8, 520, 776), (2, 6, 7, 64, 2048),
                                         (2, 64, 70, 72, 136), (2, 65, 70, 64, 64)])
def test_several_rows_at_a_time_give_the_bits_of_one(T, top, E, D, F, gated, block):
    """Inputs that do not start on 16 bytes take the kernel of one row at a time: remainders of every unrolled step, outputs that
    the last warps do not have, 48 KB of inputs, identity experts, one choice more than the kernel holds."""
    from longbow_quarrel_b200.kernels import ops
    g = torch.Generator().manual_seed(T + D + F)
    draw = lambda *n: torch.randn(n, generator=g)
    h, w_up = draw(T, D).to(torch.bfloat16).to(DEV), (draw(E, F * (2 if gated else 1), D) / D ** 0.5).to(torch.bfloat16).to(DEV)
    w_down = (draw(E, D, F) / F ** 0.5).to(torch.bfloat16).to(DEV)
    ids = torch.stack([torch.randperm(E + 2, generator=g)[:top] for _ in range(T)]).to(torch.int32).to(DEV)
    weights = torch.rand(T, top, generator=g).to(DEV)
    off = lambda t: torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)[1:].view(t.shape).copy_(t)
    u, u_one = (ops.moe_up(rows, w_up, ids, "silu", gated=gated, block=block) for rows in (h, off(h)))
    real = ids < E
    assert torch.equal(u[real], u_one[real])
    rows = w_up.double().cpu()
    if gated and block:
        rows = rows.view(E, F // 8, 2, 8, D).transpose(1, 2).reshape(E, 2 * F, D)
    pre = torch.einsum("tjfd,td->tjf", rows[ids.cpu().clamp(max=E - 1).long()], h.double().cpu())
    want = torch.nn.functional.silu(pre[..., :F]) * (pre[..., F:] if gated else 1)
    # half a unit of bfloat16; the sums' roundings: D products of about 1 / sqrt(D)
    assert bool(((u.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5)[real.cpu()].all())
    u = torch.where(real[..., None], u, torch.zeros((), dtype=u.dtype, device=DEV))
    shared, z = draw(T, D).to(DEV), draw(T, 3).to(DEV)
    for accumulate in (False, True):
        x = [torch.ones(T, D, device=DEV) for _ in range(2)]
        for into, rows in zip(x, (u, off(u))):
            ops.moe_down(rows, w_down, ids, weights, into, accumulate, shared, z[:, 1], h=h)
        assert torch.equal(x[0], x[1])
    ops.check_status()
