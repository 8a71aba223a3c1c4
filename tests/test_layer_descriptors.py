"""Descriptors of the functional interface are kept by value: what a call describes is what its arguments are worth at the call."""
import math

import numpy as np
import pytest
import torch

from smallframework_b200 import interface as S

FIELDS = (2, 16, 32, 9, 7, 3, 3, 1, 1, 1, 1, 1, 0, S.ACT_LEAKY, 0.25, -128, -121, 0, 7, 1 << 30, 0)


def described(**changed):
    names = [n for n, _ in S.Layer._fields_][:len(FIELDS)]
    ref, ho, wo = S._described(*[changed.get(n, v) for n, v in zip(names, FIELDS)])
    return ref._obj, ho, wo


def test_fields_and_output_size():
    L, ho, wo = described()
    assert tuple(getattr(L, n) for n, _ in S.Layer._fields_) == FIELDS + (0,) and (ho, wo) == (9, 7)
    assert described()[0] is L  # kept


def test_slopes_of_either_zero():
    assert math.copysign(1, described(slope=0.0)[0].slope) == 1
    assert math.copysign(1, described(slope=-0.0)[0].slope) == -1
    assert math.isnan(described(slope=float("nan"))[0].slope)


@pytest.mark.parametrize("dim", [torch.tensor(9), np.array(9)], ids=["tensor", "array"])
def test_a_dimension_that_is_written_to(dim):
    assert described(H=dim)[0].H == 9
    dim += 2
    L, ho, _ = described(H=dim)
    assert L.H == 11 and ho == 11


def test_what_a_descriptor_refuses():
    with pytest.raises(TypeError):
        described(H=9.0)
    assert described(slope=1e300)[0].slope == math.inf
