"""Calls of 2^31 evaluations and more, whose places no longer fit the products that smaller calls are divided by."""
import pytest
import torch

from hingetreefortorch_b200 import _cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner", [(), (3,)])
def test_leaf_map_of_more_than_two_to_the_31_evaluations(inner):
    T, C, K = 64, 2, 3 if inner else 1
    B = 2 ** 31 // (T * K) + 1
    generator = torch.Generator("cuda").manual_seed(0)
    x = torch.randn((B, C) + inner, generator=generator, device="cuda")
    thr = torch.randn((T, 1), generator=generator, device="cuda")
    ord_ = torch.randint(0, C, (T, 1), generator=generator, device="cuda")
    f = _cabi.Forest("tree", x, torch.empty((T, 2), device="cuda"), backward_workspace=False)
    leaf = f.leafmap(x, thr, ord_)
    assert leaf.numel() > 2 ** 31
    bounds = thr.reshape((T,) + (1,) * len(inner))
    for first in range(0, B, 1 << 20):
        rows = slice(first, min(first + (1 << 20), B))
        assert torch.equal(leaf[rows], (x[rows].index_select(1, ord_[:, 0]) > bounds).long())
    assert f.ordinal_flags() == 0
