"""What a step's tokens may be: whole numbers of any kind, as torch reads them, and nothing that merely looks like one."""
from decimal import Decimal

import numpy as np
import pytest
import torch

from citlali_b200.engine.step import StepEntry, pack_step

CPU = torch.device("cpu")


def packed(tokens):
    return pack_step([StepEntry(0, tokens, [len(tokens) - 1])], [3], 100, CPU).tokens.tolist()


@pytest.mark.parametrize("tokens", [
    [1, 2, 99], (1, 2, 99), np.array([1, 2, 99]), np.array([1, 2, 99], dtype=np.uint8), [np.int32(1), 2, np.uint64(99)],
    torch.tensor([1, 2, 99]), [torch.tensor(1), torch.tensor(2), 99], [True, 2, 99], [1.0, 2.0, 99.0], range(1, 100, 49)], ids=repr)
def test_numbers_are_tokens(tokens):
    want = [1, 50, 99] if isinstance(tokens, range) else [1, 2, 99]
    assert packed(tokens) == want == torch.as_tensor(list(tokens), dtype=torch.int64).tolist()


@pytest.mark.parametrize("tokens", [["5"], [1, "5"], [np.str_("5"), 6], "55", [None], [Decimal(5)], [1 + 0j], [float("nan")],
                                    [2 ** 63], [2 ** 70], [np.datetime64(5, "s")], [[1], [2]], [[1], [2, 3]]], ids=repr)
def test_what_torch_does_not_read_is_refused(tokens):
    with pytest.raises(Exception):
        packed(tokens)


@pytest.mark.parametrize("tokens", [[-1], [100], [5, 2 ** 40], [-2 ** 63]])
def test_tokens_outside_the_vocabulary_are_named(tokens):
    with pytest.raises(Exception, match=rf"token id {tokens[-1]} out of vocab range \[0, 100\)"):
        packed(tokens)
