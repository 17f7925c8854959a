"""The tables of words that calls pass to the library take whatever holds whole numbers: lists, tuples, tensors and
arrays of any numeric type, and floats, which are truncated."""
import numpy as np
import pytest
import torch

from proving_gb300.backend import _u32_table

WORDS = [0, 1, 77, (1 << 31) - 2]


@pytest.mark.parametrize("make", [list, tuple, torch.tensor, np.array, lambda w: np.array(w, np.uint32), lambda w: np.array(w, np.float64),
                                  lambda w: np.array(w, object), lambda w: [float(x) + 0.5 for x in w]])
def test_words(make):
    assert list(_u32_table(make(WORDS))) == WORDS


def test_no_words_and_wrapped_words():
    assert len(_u32_table([])) == 1 and len(_u32_table(np.array([], np.uint32))) == 1
    assert list(_u32_table([-1, 1 << 32])) == [0xffffffff, 0] and list(_u32_table(np.array([-1]))) == [0xffffffff]
