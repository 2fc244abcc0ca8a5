"""A step's tokens as one array: the same packing and the same errors as lists looked at one by one."""

import numpy as np
import pytest
import torch

from longbow_quarrel_b200.engine.step import StepError, check_entries, pack_step, whole

L = list(range(20))


@pytest.mark.parametrize("tokens", [[5], L, tuple(L), L[:15], L[:16], np.arange(20), torch.arange(20), [np.int32(3)] * 20, [torch.tensor(3)] * 20,
                                    L + [True], L + [3.7], L + [-0.5], L + [100], L + [-1], L + [2 ** 70], L + ["x"], L + [None],
                                    L + [float("nan")], [], np.arange(20) + 90, np.arange(40).reshape(20, 2)])
def test_a_list_made_whole_is_taken_or_refused_as_the_list_itself(tokens):
    def outcome(t):
        try:
            check_entries([(0, t)], None, 100)
            return pack_step([(0, t)], None, [3], {})[0].tolist()
        except Exception as error:
            return type(error), str(error)
    assert outcome(whole(tokens)) == outcome(tokens)


def test_the_first_token_outside_is_named():
    with pytest.raises(StepError, match=r"token 100 at place 20 of sequence 0 is outside the vocabulary \[0, 100\)"):
        check_entries([(0, whole(L + [100, -1]))], None, 100)
