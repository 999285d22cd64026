"""The base tables that a paged attention call is given: a sequence of four or more, of which the first four count."""
import pytest
import torch
from test_split_rules import calls, _paged


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("bases", [(1, 2, 3, 4), [1, 2, 3, 4, 5], {i: i + 1 for i in range(4)}, torch.arange(1, 6)])
def test_the_first_four_tables(calls, bases, wide):
    name, a = _paged(calls, 1, 2, 4, 4, wide, bases)
    assert len(a[0]) == 13 and [int(t) for t in a[0][6:10]] == [1, 2, 3, 4]


def test_fewer_are_refused(calls):
    with pytest.raises(IndexError): _paged(calls, 1, 2, 4, 4, False, (1, 2, 3))
