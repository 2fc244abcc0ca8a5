"""Latent attention of prompts over expanded keys and values (csrc/latent_prefill.cu) against the same part in 32-bit and against
its absorbed form: edges of the 128-row chains and 128-key tiles, portions, windows, a sink, sequences side by side."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
D, R = 192, 64


def _part(dtype, H, window, sink, weights=None, scale=0.12):
    from longbow_quarrel_b200.parts.base import Runtime
    from longbow_quarrel_b200.parts.latent_attention import LatentAttention
    from longbow_quarrel_b200.parts.spec import PartSpec
    from longbow_quarrel_b200.weights import random_weights
    part = LatentAttention(Runtime(DEV, dtype, 2048), hidden_size=D, n_heads=H, head_dim=128, rot_dim=64, value_dim=128, q_rank=None, kv_rank=R,
                           scale=scale, eps=1e-5, position=PartSpec("rope", {"head_dim": 64, "theta": 1e4}), window=window, sink=sink)
    weights = weights or random_weights(part.weights(), 3, torch.bfloat16, DEV, std=0.08)
    part.load(weights)
    return part, weights


def _run(part, portions, h):
    """Steps of the sequences, portion by portion: the rows of every sequence, in order."""
    from longbow_quarrel_b200.cache import Cache
    from longbow_quarrel_b200.engine.step import make_context, pack_step
    from longbow_quarrel_b200.kernels import ops
    cache = Cache({0: part.cache_need()}, 8192, 2048, part.runtime.dtype, DEV, max_slots=4)
    slots = [cache.alloc_slot() for _ in h]
    past, got, routes = [0] * len(h), [[] for _ in h], []
    for step in portions:
        live = [i for i, n in enumerate(step) if n]
        for i in live:
            cache.reserve(slots[i], step[i])
        cache.upload()
        flat, info = pack_step([(slots[i], [0] * step[i]) for i in live], None, [past[i] for i in live], part.step_needs())
        ctx = make_context(torch.from_numpy(flat).to(DEV), info, [slots[i] for i in live])
        rows = torch.cat([h[i][past[i]:past[i] + step[i]] for i in live]).to(part.runtime.dtype)
        before = ops.launches_by_name().get("latent_prefill", 0)
        out = part.forward(rows, ctx, cache.view(0), None)
        routes.append(ops.launches_by_name().get("latent_prefill", 0) - before)
        at = 0
        for i in live:
            got[i].append(out[at:at + step[i]])
            at += step[i]
            past[i] += step[i]
            cache.commit(slots[i], step[i])
    torch.cuda.synchronize()
    ops.check_status()
    return [torch.cat(g).double() for g in got], routes


@pytest.mark.parametrize("H,window,sink,portions", [
    (2, None, False, [(128,)]), (3, None, True, [(129, 257, 40)]), (2, None, False, [(300, 0), (70, 511), (33, 100)]), (1, 100, True, [(450, 130), (200, 64)]),
    (2, 300, False, [(700,), (129,)]), (16, None, False, [(1100,)]),
    (16, None, True, [(1300, 1290)])])           # the last: more blocks than multiprocessors, whose chains are neighbours (2 i, 2 i + 1)
def test_expanded_prompts_agree_with_32_bit_and_with_the_absorbed_form(H, window, sink, portions, monkeypatch):
    from longbow_quarrel_b200.kernels import attention as kernels
    gen = torch.Generator().manual_seed(H)
    h = [torch.randn(sum(s[i] for s in portions), D, generator=gen).to(torch.bfloat16).to(DEV) for i in range(len(portions[0]))]
    part, weights = _part(torch.bfloat16, H, window, sink)
    got, routes = _run(part, portions, h)
    assert all(routes)
    monkeypatch.setattr(kernels, "EXPAND_QUERIES", 10 ** 9)
    absorbed, routes = _run(part, portions, h)
    assert not any(routes)
    want, _ = _run(_part(torch.float32, H, window, sink, weights)[0], portions, h)
    for g, a, w in zip(got, absorbed, want):
        err, other = float((g - w).norm() / w.norm()), float((a - w).norm() / w.norm())
        # Both forms round three tensors to bfloat16 on the way (2^-9 each at most, at random); neither may lose against the other (of
        # the attention alone, over 2 to 32 heads and latents of 64 to 512, their distances from 64 bits differ by 4 % at most, either way).
        assert err < 3 * 2.0 ** -8 and err < 1.1 * other, (err, other)
        assert float((g - w).abs().max()) < 0.06 * float(w.abs().max())


@pytest.mark.parametrize("H,window,portions,expanded", [
    (2, None, [(200, 600, 5), (1, 1, 1), (1, 130, 9)], [1, 0, 1]), (16, None, [(700, 300), (1, 33)], [1, 1]), (3, 90, [(9, 260, 1), (40, 7, 15)], [1, 1])])
def test_a_step_of_long_and_short_portions_runs_in_both_forms(H, window, portions, expanded):
    gen = torch.Generator().manual_seed(H)
    h = [torch.randn(sum(s[i] for s in portions), D, generator=gen).to(torch.bfloat16).to(DEV) for i in range(len(portions[0]))]
    part, weights = _part(torch.bfloat16, H, window, True)
    got, routes = _run(part, portions, h)
    assert routes == expanded
    want, _ = _run(_part(torch.float32, H, window, True, weights)[0], portions, h)
    for g, w in zip(got, want):
        assert float((g - w).norm() / w.norm()) < 3 * 2.0 ** -8 and float((g - w).abs().max()) < 0.06 * float(w.abs().max())


def test_sequences_in_turns(monkeypatch):
    """Buffers that hold two of the four sequences: the same result as all at once, bit for bit."""
    from longbow_quarrel_b200.kernels import attention as kernels
    gen = torch.Generator().manual_seed(9)
    h = [torch.randn(n, D, generator=gen).to(torch.bfloat16).to(DEV) for n in (300, 200, 270, 1)]
    part, _ = _part(torch.bfloat16, 2, None, False)
    want, routes = _run(part, [(300, 200, 270, 1)], h)
    assert routes == [1]
    monkeypatch.setattr(kernels, "EXPAND_ELEMENTS", 500 * (2 * 256 + R + 64))
    got, routes = _run(part, [(300, 200, 270, 1)], h)
    assert routes == [2] and all(torch.equal(g, w) for g, w in zip(got, want))


def test_no_memory_for_the_expansion(monkeypatch):
    from longbow_quarrel_b200.kernels import ops
    gen = torch.Generator().manual_seed(4)
    h = [torch.randn(n, D, generator=gen).to(torch.bfloat16).to(DEV) for n in (200, 3)]
    part, weights = _part(torch.bfloat16, 2, None, True)

    def full(*args):
        raise torch.cuda.OutOfMemoryError("test")
    monkeypatch.setattr(ops, "latent_gather", full)
    got, routes = _run(part, [(200, 3)], h)
    assert routes == [0]
    want, _ = _run(_part(torch.float32, 2, None, True, weights)[0], [(200, 3)], h)
    for g, w in zip(got, want):
        assert float((g - w).norm() / w.norm()) < 3 * 2.0 ** -8


def test_few_queries_per_key_keep_the_absorbed_form():
    gen = torch.Generator().manual_seed(1)
    part, weights = _part(torch.bfloat16, 2, None, False)
    h = [torch.randn(310, D, generator=gen).to(torch.bfloat16).to(DEV)]
    got, routes = _run(part, [(300,), (9,), (1,)], h)
    assert routes == [1, 0, 0]
    want, _ = _run(_part(torch.float32, 2, None, False, weights)[0], [(310,)], h)
    assert float((got[0] - want[0]).norm() / want[0].norm()) < 3 * 2.0 ** -8


@pytest.mark.parametrize("H,window,portions,spoiled", [
    (2, None, [(100, 70)], (0, 60)), (2, None, [(100, 70)], (1, 0)), (1, None, [(300, 40), (20, 200)], (0, 130)), (2, 90, [(400, 200)], (0, 137)),
    (16, None, [(700, 31)], (0, 699))])
def test_a_row_that_is_not_finite_spoils_only_the_rows_that_see_it(H, window, portions, spoiled):
    """A token of NaN: every row that sees it is NaN, and no other, ahead of it in its sequence or in its neighbour, whose expanded rows
    share a tile of keys with it."""
    gen = torch.Generator().manual_seed(5)
    h = [torch.randn(sum(s[i] for s in portions), D, generator=gen).to(torch.bfloat16).to(DEV) for i in range(len(portions[0]))]
    part, _ = _part(torch.bfloat16, H, window, False)
    clean, _ = _run(part, portions, h)
    h[spoiled[0]][spoiled[1]] = float("nan")
    got, routes = _run(part, portions, h)
    assert all(routes)
    for i, (g, c) in enumerate(zip(got, clean)):
        at = torch.arange(g.shape[0], device=DEV)
        sees = (at >= spoiled[1]) & ((at < spoiled[1] + window) if window else True) & (i == spoiled[0])
        assert torch.isnan(g[sees]).all() and torch.equal(g[~sees], c[~sees])


@pytest.mark.parametrize("scale", [-0.12, 0.0])
def test_scales_that_are_not_positive_keep_the_absorbed_form(scale):
    gen = torch.Generator().manual_seed(2)
    h = [torch.randn(150, D, generator=gen).to(torch.bfloat16).to(DEV)]
    part, weights = _part(torch.bfloat16, 2, None, False, scale=scale)
    got, routes = _run(part, [(150,)], h)
    assert routes == [0]
    want, _ = _run(_part(torch.float32, 2, None, False, weights, scale=scale)[0], [(150,)], h)
    assert float((got[0] - want[0]).norm() / want[0].norm()) < 3 * 2.0 ** -8
