"""The plain attention kernel (csrc/plain_kernels.cu) where its cached rows lie far out."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def test_pages_behind_two_to_the_31st_row():
    """8.6 GB of pages of heads of two: a sequence in the last pages has the result that it has in the first ones."""
    from longbow_quarrel_b200.kernels import ops
    page, hd, n = 64, 2, 130
    last = 2 ** 31 // page
    pages = torch.empty((last + 3, 1, page, hd), dtype=torch.bfloat16, device=DEV)
    gen = torch.Generator().manual_seed(1)
    rows = torch.randn(3, 1, page, hd, generator=gen).to(torch.bfloat16).to(DEV)
    q = torch.randn(2, hd, generator=gen).to(torch.bfloat16).to(DEV)
    pages[last:] = rows
    pages[:3] = rows
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table = torch.tensor([[0, 1, 2], [last, last + 1, last + 2]], dtype=torch.int32, device=DEV)
    run = lambda slot: ops.attention_plain(q, pages, pages, table, i32(n - 2, n - 1), i32(0, 0), i32(slot), 1, 1, hd, page, 0.5, None)
    near, far = run(0), run(1)
    keys = rows.reshape(-1, hd).double()
    want = torch.stack([torch.softmax(keys[:m] @ x.double() * 0.5, 0) @ keys[:m] for m, x in zip((n - 1, n), q)])
    assert torch.equal(near, far)
    assert float((near.double() - want).abs().max()) < 2.0 ** -8 * float(want.abs().max())      # bfloat16 results
