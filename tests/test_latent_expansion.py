"""Which steps expand latent keys and values, and the work list of those that do (host logic only)."""
import numpy as np
import pytest

from longbow_quarrel_b200.kernels.attention import EXPAND_QUERIES, EXPAND_TILE, expanded_rows, expanded_work, expands
from longbow_quarrel_b200.parts.base import StepShape


def _step(past, new):
    cu = tuple(int(c) for c in np.concatenate([[0], np.cumsum(new)]))
    return StepShape(B=len(new), T=cu[-1], past=tuple(past), new=tuple(new), cu=cu)


@pytest.mark.parametrize("past,new,window,expected", [
    ((0,), (1,), 0, False), ((0, 50), (1, 1), 0, False), ((0,), (EXPAND_QUERIES,), 0, True), ((0,), (EXPAND_QUERIES - 1,), 0, False),
    ((4000,), (10,), 0, False), ((4000,), (100,), 0, True), ((0, 4000), (200, 1), 0, False), ((0, 4000), (200, 1), 128, True)])
def test_steps_with_enough_queries_per_key_expand(past, new, window, expected):
    assert expands(past, new, window, 16, 256) is expected
    assert (len(expanded_work(16, 256, window, 148)(_step(past, new))) > 0) is expected


@pytest.mark.parametrize("past,new,window", [((0,), (500,), 0), ((0, 130, 7), (128, 700, 129), 0), ((300,), (1000,), 100), ((90, 1000), (257, 65), 300)])
@pytest.mark.parametrize("sms", [2, 148])
def test_every_row_is_in_one_chain_and_every_key_it_sees_among_its_tiles(past, new, window, sms):
    step = _step(past, new)
    flat = expanded_work(2, 256, window, sms)(step)
    B = step.B
    n = (len(flat) - 2 * B - 1) // 7
    blocks, first_row, lo = flat[:7 * n].reshape(7, n).T, flat[7 * n:7 * n + B + 1], flat[7 * n + B + 1:]
    assert lo.tolist() == expanded_rows(past, new, window)[0] and np.diff(first_row).tolist() == expanded_rows(past, new, window)[1]
    seen = np.zeros(step.T, dtype=int)
    for b, *chains in blocks:
        spans = []
        for row, rows, pos in (chains[:3], chains[3:]):
            if rows == 0:
                continue
            assert 1 <= rows <= 128 and step.cu[b] <= row and row + rows <= step.cu[b + 1] and pos - past[b] == row - step.cu[b]
            seen[row:row + rows] += 1
            first = max(0, pos - window + 1) if window else 0
            assert first >= lo[b] and lo[b] % EXPAND_TILE == 0
            spans.append((first // EXPAND_TILE, (pos + rows - 1) // EXPAND_TILE + 1))
        assert spans and chains[1] > 0
        if len(spans) == 2:                    # the tiles that a block walks have no gap
            assert max(s[0] for s in spans) <= min(s[1] for s in spans)
    assert (seen == 1).all()
    work = [sum((e[k + 2] + e[k + 1]) // 128 + 1 for k in (1, 4) if e[k + 1]) for e in blocks]
    assert work == sorted(work, reverse=True)
