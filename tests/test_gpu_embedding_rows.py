"""The embedding of whole eights of columns: the table's numbers, whichever kernel reads them."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,V,D,scale", [(1, 3, 8, 1.0), (7, 50, 2040, 0.7), (3, 50, 2056, 1.0), (300, 1000, 4096, 1.3), (5, 9, 20, 0.7)])
def test_rows_of_the_table_times_the_scale(dtype, T, V, D, scale):
    """One vector, a block's 2,048 columns less and plus one vector, two rounds, and a width and a start that no vector allows."""
    from longbow_quarrel_b200.kernels import ops
    g = torch.Generator().manual_seed(D)
    table = torch.randn(V, D, generator=g).to(dtype).to(DEV)
    tokens = torch.randint(0, V, (T,), generator=g).to(torch.int32).to(DEV)
    want = table[tokens.long()].float() * scale
    assert torch.equal(ops.embedding(table, tokens, scale=scale), want)
    off = torch.empty(V * D + 1, dtype=dtype, device=DEV)[1:].view(V, D).copy_(table)
    assert torch.equal(ops.embedding(off, tokens, scale=scale), want)
