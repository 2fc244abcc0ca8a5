"""What surrounds the experts' products of a prompt: the pairs' order by groups, the rows' gather, their combination."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _ops():
    from longbow_quarrel_b200.kernels import ops

    return ops


@pytest.mark.parametrize("n,G", [(1, 1), (128, 1), (129, 2), (1023, 31), (1025, 33), (6000, 64), (4096, 1000), (5, 6144)])
def test_every_index_has_one_place_in_a_tile_of_its_group(n, G):
    """Around one warp's sum of the groups' tiles (32 at a time) and the 1024 threads; empty groups first, between and last; ids at
    G and above have no place."""
    ops = _ops()
    g = torch.Generator().manual_seed(n + G)
    used = torch.randperm(G, generator=g)[:max(1, G * 2 // 3)]
    ids = used[torch.randint(0, len(used), (n,), generator=g)].to(torch.int32)
    if n > 1000:
        ids[::7] = G + 3
    src, dst, tile_group = (t.cpu().long() for t in ops.group_rows_padded(ids.to(DEV), G))
    flat = ids.long()
    placed = flat < G
    assert (dst[~placed] == -1).all() and (src[dst[placed]] == torch.arange(n)[placed]).all()
    assert int((src >= 0).sum()) == int(placed.sum())
    tiles = (torch.bincount(flat[placed], minlength=G) + 127) // 128
    want = torch.cat([torch.repeat_interleave(torch.arange(G), tiles), torch.full((len(tile_group) - int(tiles.sum()),), -1)])
    assert (tile_group == want).all() and (tile_group[dst[placed] // 128] == flat[placed]).all()
    h = torch.randn(n, 8, generator=g).to(torch.bfloat16)
    rows = ops.gather_rows(h.to(DEV), src.to(torch.int32).to(DEV), 1, tile_group.to(torch.int32).to(DEV)).cpu()
    inside = torch.repeat_interleave(tile_group >= 0, 128)
    assert torch.equal(rows[inside], torch.where((src >= 0)[:, None], h[src.clamp(min=0)], 0.0)[inside])
    ops.check_status()


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("T,top,D,identity", [(3, 1, 4, False), (17, 6, 104, True), (5, 8, 1028, False), (2, 64, 256, True), (2, 65, 256, False)])
def test_the_combination_of_four_columns_at_a_time_is_that_of_one(T, top, D, identity, accumulate):
    """The same products in the same order: rows that do not start on 16 bytes take the other kernel, with the same bits."""
    ops = _ops()
    g = torch.Generator().manual_seed(T + D)
    y = torch.randn(T * top, D, generator=g).to(DEV)
    h = torch.randn(T, D, generator=g).to(torch.bfloat16).to(DEV)
    weights = torch.rand(T, top, generator=g).to(DEV)
    shared, z = torch.randn(T, D, generator=g).to(DEV), torch.randn(T, 3, generator=g).to(DEV)
    place = torch.randperm(T * top, generator=g).to(torch.int32).to(DEV)
    ids = torch.randint(0, 9, (T, top), generator=g).to(torch.int32).to(DEV)
    more = dict(ids=ids, E=7, h=h) if identity else {}
    x = torch.randn(T, D, generator=g).to(DEV)
    off = torch.empty(T * D + 1, device=DEV)[1:].view(T, D).copy_(x)
    for into in (x, off):
        ops.moe_combine(y, weights, into, accumulate, shared=shared, shared_gate=z[:, 2], place=place, shared_scale=0.5, **more)
    assert torch.equal(x, off)
    ops.check_status()


@pytest.mark.parametrize("T,E,D,F", [(130, 3, 64, 8), (300, 5, 128, 264), (140, 2, 520, 136)])
@pytest.mark.parametrize("act", ["gelu", "gelu_tanh", "silu", "relu", "relu2"])
def test_a_grouped_product_behind_an_activation(act, T, E, D, F):
    """The activation of the float32 sums ahead of their one rounding: the product's own float32 output, activated in 64 bits, at
    widths of one vector, of a tile and one vector more, and of half a tile."""
    ops = _ops()
    g = torch.Generator().manual_seed(T + F)
    h = torch.randn(T, D, generator=g).to(torch.bfloat16).to(DEV)
    w = (2 * torch.randn(E, F, D, generator=g) / D ** 0.5).to(torch.bfloat16).to(DEV)
    ids = torch.randint(0, E, (T,), generator=g).to(torch.int32).to(DEV)
    src, dst, tile_group = ops.group_rows_padded(ids, E)
    rows = ops.gather_rows(h, src, 1, tile_group)
    sums = ops.gemm_tc_grouped(rows, w, tile_group, torch.float32)[dst.long()].double()
    got = ops.gemm_tc_grouped(rows, w, tile_group, torch.bfloat16, act=act)[dst.long()].double()
    want = {"gelu": lambda v: 0.5 * v * (1 + torch.erf(v / 2 ** 0.5)), "silu": lambda v: v * torch.sigmoid(v), "relu": torch.relu,
            "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh"), "relu2": lambda v: torch.relu(v) ** 2}[act](sums)
    # half a unit of bfloat16, and a few float32 roundings of the factor (1 + erf or tanh), which cancels for negative sums
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 16 * 2.0 ** -24 * sums.abs()).all())
    ops.check_status()


@pytest.mark.parametrize("groups", [[0], [0, 0, 0, -1], [1, 1, 2, 2, 2, 3, -1, -1], [3, 3, 0, 0, 0, -1, 3, 1, -1, 1], list(range(5)) * 2 + [4] * 160])
@pytest.mark.parametrize("N,K", [(8, 64), (600, 72), (8, 3072), (600, 3080)])      # tiles by row tiles, then by groups
def test_grouped_products_walk_every_tile_once_in_whatever_order_the_groups_come(groups, N, K):
    """One to three columns of tiles, runs of one group and groups that come back; more tiles than multiprocessors.  Integers small enough
    that every sum is exact."""
    ops = _ops()
    g = torch.Generator().manual_seed(len(groups))
    a = torch.randint(-3, 4, (len(groups) * 128, K), generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randint(-3, 4, (5, N, K), generator=g).to(torch.bfloat16).to(DEV)
    tiles = torch.tensor(groups, dtype=torch.int32, device=DEV)
    got = ops.gemm_tc_grouped(a, w, tiles, torch.float32).view(len(groups), 128, N)
    for i, group in enumerate(groups):
        if group >= 0:
            assert torch.equal(got[i], (a[i * 128:(i + 1) * 128].float() @ w[group].float().T))
    ops.check_status()
