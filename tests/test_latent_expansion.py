"""Which sequences of a step expand latent keys and values, and the work lists of both forms (host logic only)."""
import numpy as np
import pytest

from longbow_quarrel_b200.kernels import attention as kernels
from longbow_quarrel_b200.kernels.attention import (EXPAND_ELEMENTS, EXPAND_QUERIES, EXPAND_TILE, absorbed_rest, expanded_blocks, expanded_rows,
                                                    expanded_turns, expanded_work)
from longbow_quarrel_b200.parts.base import StepShape


def _step(past, new):
    cu = tuple(int(c) for c in np.concatenate([[0], np.cumsum(new)]))
    return StepShape(B=len(new), T=cu[-1], past=tuple(past), new=tuple(new), cu=cu)


def _turns(flat, new, turns):
    """The step array's parts: (blocks [n, 7], first rows, positions of the first rows) of every turn."""
    at, B = 0, len(new)
    for turn in turns:
        n = expanded_blocks(new, turn)
        yield flat[at:at + 7 * n].reshape(7, n).T, flat[at + 7 * n:at + 7 * n + B + 1], flat[at + 7 * n + B + 1:at + 7 * n + 2 * B + 1]
        at += 7 * n + 2 * B + 1
    assert at == len(flat)


@pytest.mark.parametrize("past,new,window,expected", [
    ((0,), (1,), 0, []), ((0, 50), (1, 1), 0, []), ((0,), (EXPAND_QUERIES,), 0, [[0]]), ((0,), (EXPAND_QUERIES - 1,), 0, []),
    ((4000,), (10,), 0, []), ((4000,), (100,), 0, [[0]]), ((0, 4000), (200, 1), 0, [[0]]), ((4000, 0), (1, 200), 128, [[1]]),
    ((0, 9, 70, 3), (16, 15, 40, 1), 0, [[0, 2]])])
def test_a_sequence_expands_by_its_own_rows(past, new, window, expected):
    assert expanded_turns(past, new, window, 16, 256, 512) == expected
    assert (len(expanded_work(16, 256, 512, window, 148)(_step(past, new))) > 0) is bool(expected)


def test_more_than_the_buffers_hold_goes_in_turns_and_a_portion_on_a_longer_past_stays_absorbed(monkeypatch):
    each = 2 * 256 + 64 + 64
    monkeypatch.setattr(kernels, "EXPAND_ELEMENTS", 1000 * each)
    assert expanded_turns((0, 0, 970, 0, 900), (400, 600, 31, 30, 100), 0, 2, 256, 64) == [[0, 1], [3], [4]]
    # A prompt has at least what the absorbed form's queries and means would take, alone in its turn.
    assert expanded_turns((0, 0, 0), (400, 5000, 300), 0, 2, 256, 64) == [[0], [1], [2]]


@pytest.mark.parametrize("H,R", [(2, 64), (16, 512), (32, 512), (128, 512)])
def test_expanded_buffers_stay_within_what_the_absorbed_form_takes_or_256_mb(H, R):
    for past, new in [((0,), (100000,)), ((0, 0, 0), (30000, 8000, 16)), ((30000,) * 40, (16,) * 40), ((100000, 500), (512, 9000)), ((10 ** 6,), (100,))]:
        _, rows = expanded_rows(past, new, 0)
        for turn in expanded_turns(past, new, 0, H, 256, R):
            bytes_ = sum(rows[b] * (H * 256 + R + 64) * 2 for b in turn)
            absorbed = sum(new[b] * H * ((R + 64) * 4 + R * 2) for b in turn)
            assert bytes_ <= max(256 << 20, absorbed)
        if past == (0,):
            assert expanded_turns(past, new, 0, H, 256, R) == [[0]]


@pytest.mark.parametrize("past,new", [((0, 4000, 5), (200, 1, 9)), ((7, 0, 30, 2), (3, 40, 15, 100)), ((0, 8), (50, 60)), ((9, 8), (1, 6)), ((100, 3), (1, 30))])
def test_the_rest_of_a_step_is_listed_for_the_absorbed_form(past, new):
    step, size = _step(past, new), 4
    flat = absorbed_rest(size, 16, 256, 512, 0)(step)
    expanded = {b for t in expanded_turns(past, new, 0, 16, 256, 512) for b in t}
    rest = [b for b in range(step.B) if b not in expanded]
    if not expanded:
        assert np.array_equal(flat, kernels.query_blocks(size)(step).reshape(-1))
        return
    T = sum(new[b] for b in rest)
    rows, blocks = flat[len(flat) - T:], flat[:len(flat) - T].reshape(4, -1).T
    assert rows.tolist() == [r for b in rest for r in range(step.cu[b], step.cu[b + 1])]
    if max((new[b] for b in rest), default=1) == 1:           # single tokens need no list
        assert len(blocks) == 0
        return
    seen = []
    for b, row, n, pos in blocks:
        assert b in rest and n <= size
        seen += [(int(b), int(rows[row + i]) - step.cu[b] + past[b], int(pos + i)) for i in range(n)]
    assert sorted(seen) == [(b, p, p) for b in rest for p in range(past[b], past[b] + new[b])]


@pytest.mark.parametrize("past,new,window", [((0,), (500,), 0), ((0, 130, 7), (128, 700, 129), 0), ((300,), (1000,), 100), ((90, 1000), (257, 65), 300)])
@pytest.mark.parametrize("sms", [2, 148])
@pytest.mark.parametrize("held", [EXPAND_ELEMENTS, 1200 * 640])
def test_every_row_is_in_one_chain_and_every_key_it_sees_among_its_tiles(past, new, window, sms, held, monkeypatch):
    monkeypatch.setattr(kernels, "EXPAND_ELEMENTS", held)
    step = _step(past, new)
    firsts, rows = expanded_rows(past, new, window)
    turns = expanded_turns(past, new, window, 2, 256, 64)
    assert sorted(b for t in turns for b in t) == list(range(step.B))
    seen, listed = np.zeros(step.T, dtype=int), []
    for turn, (blocks, first_row, lo) in zip(turns, _turns(expanded_work(2, 256, 64, window, sms)(step), new, turns)):
        assert lo.tolist() == firsts and np.diff(first_row).tolist() == [r if b in turn else 0 for b, r in enumerate(rows)]
        assert set(blocks[:, 0]) == set(turn)
        work = [sum((e[k + 2] + e[k + 1]) // 128 + 1 for k in (1, 4) if e[k + 1]) for e in blocks]
        assert work == sorted(work, reverse=True)
        listed += blocks.tolist()
    for b, *chains in listed:
        spans = []
        for row, rows, pos in (chains[:3], chains[3:]):
            if rows == 0:
                continue
            assert 1 <= rows <= 128 and step.cu[b] <= row and row + rows <= step.cu[b + 1] and pos - past[b] == row - step.cu[b]
            seen[row:row + rows] += 1
            first = max(0, pos - window + 1) if window else 0
            assert first >= firsts[b] and firsts[b] % EXPAND_TILE == 0
            spans.append((first // EXPAND_TILE, (pos + rows - 1) // EXPAND_TILE + 1))
        assert spans and chains[1] > 0
        if len(spans) == 2:                    # the tiles that a block walks have no gap
            assert max(s[0] for s in spans) <= min(s[1] for s in spans)
    assert (seen == 1).all()


def test_matrices_that_are_views_of_one_another_are_weighed_once():
    import torch

    from longbow_quarrel_b200.engine.model import Model

    class Part:
        def __init__(self):
            self.both = torch.zeros(6, 4)
            self.first, self.second, self.other = self.both[:2].view(1, 2, 4), self.both[2:], torch.zeros(3, dtype=torch.bfloat16)

    model = object.__new__(Model)
    part = Part()
    model._named_parts = lambda: [("a", part), ("b", part)]
    assert model.weight_bytes() == 6 * 4 * 4 + 3 * 2
