"""Several outputs per leaf: rows of every width the kernels distinguish, tiles of evaluations that end anywhere, inner
positions, both ways to the paths (kept by the forward, or walked again)."""
import numpy as np
import pytest
import torch

import hingetreefortorch_b200._cabi as _cabi
from conftest import grad_close
from oracle import hinge_oracle as ho
from test_forest_gpu import dev, random_forest_inputs

pytestmark = pytest.mark.gpu

# B, C, inner, T, depth, M: evaluations per tree around multiples of 1024; pieces of one, two and four numbers per row, up
# to one lane, half a warp and a whole warp of them; one level and twelve
SHAPES = [
    (1025, 9, (), 40, 3, 2),
    (1024, 300, (), 33, 4, 3),
    (2047, 20, (), 17, 12, 4),
    (1500, 8, (), 30, 1, 5),
    (300, 31, (7,), 21, 6, 6),
    (999, 16, (), 37, 9, 7),
    (3, 50, (41, 25), 12, 5, 8),
    (1100, 40, (), 31, 10, 10),
    (1, 12, (1023,), 35, 7, 17),
    (2100, 64, (), 16, 8, 26),
    (513, 11, (2,), 33, 4, 33),
    (5, 16, (900,), 9, 11, 63),
    (2, 100, (24, 24), 30, 7, 64),
    # many features: the walk goes row by row (last rows not a whole step; groups of trees; two trees' worth of outputs per lane)
    (1003, 333, (), 40, 5, 10),
    (1001, 784, (), 48, 5, 3),
    (2050, 784, (), 300, 8, 1),
    (8195, 200, (), 4, 3, 2),
    # leaf weights that do not fit beside a tile; few trees whose samples are split among blocks
    (9500, 719, (), 6, 12, 1),
    (9000, 30, (), 4, 10, 1),
    (33000, 12, (), 3, 4, 1),
    # too few evaluations for the sorted backward, but not for the fixed order; one output, more than a buffer of terms holds
    (31, 5, (), 3, 2, 2),
    (700, 20, (), 6, 7, 1),
    (130, 9, (5,), 2, 3, 70),
    (3, 4, (), 2, 1, 4500),
]


@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("shape", SHAPES, ids=[str(s) for s in SHAPES])
def test_forward_and_backward(kind, shape):
    B, C, inner, T, depth, M = shape
    x, thr, ord_, w = random_forest_inputs(300 + SHAPES.index(shape), kind, B, C, inner, T, depth, (M,), quantise=True)
    want = ho.forward(kind, x, thr, ord_, w)
    g = np.random.default_rng(5).standard_normal(want.shape).astype(np.float32)
    ref = ho.backward(kind, x, thr, ord_, w, g)
    sizes = ho.backward_magnitudes(kind, x, thr, ord_, w, g)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    f = _cabi.Forest(kind, dx, dw)
    for got, r, s in zip(f.backward(dx, dthr, dord, dw, dg), ref, sizes):
        assert grad_close(got, r, s)
    only_thr = f.backward(dx, dthr, dord, dw, dg, need=(False, True, False))
    assert only_thr[0] is None and grad_close(only_thr[1], ref[1], sizes[1]) and only_thr[2] is None
    assert np.array_equal(f.forward(dx, dthr, dord, dw, save=True).cpu().numpy(), want)
    for got, r, s in zip(f.backward(dx, dthr, dord, dw, dg, saved=True), ref, sizes):
        assert grad_close(got, r, s)
    ordered = _cabi.Forest(kind, dx, dw, deterministic=True)
    for got, r in zip(ordered.backward(dx, dthr, dord, dw, dg), ref):
        assert np.array_equal(got.cpu().numpy(), r)
    assert np.array_equal(ordered.forward(dx, dthr, dord, dw, save=True).cpu().numpy(), want)
    for got, r in zip(ordered.backward(dx, dthr, dord, dw, dg, saved=True), ref):
        assert np.array_equal(got.cpu().numpy(), r)
    x.reshape(-1)[:3] = [np.inf, -np.inf, np.nan]
    got = f.forward(dev(x)[0], dthr, dord, dw).cpu().numpy()
    assert np.array_equal(got, ho.forward(kind, x, thr, ord_, w), equal_nan=True)
    assert f.ordinal_flags() == 0


# evaluations per tree around whole slices (960 with three or five lanes per row, 1024 otherwise), leaves that a few or all
# evaluations share, samples that begin inside a slice; pieces of one, two and four numbers, listed rows and others
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("M", [2, 3, 5, 10, 12, 20, 26, 32, 64])
@pytest.mark.parametrize("B, inner, depth", [(959, (), 7), (960, (), 1), (961, (), 9), (1024, (), 2), (1025, (), 8), (1923, (), 4),
                                             (7, (11, 25), 5)])
def test_slices_of_the_sorted_backward(B, inner, depth, M, dtype):
    T, C = -(-32768 // (B * int(np.prod(inner, dtype=int)))) + 1, 10
    kind = "tree" if M % 2 == 0 else "fern"
    x, thr, ord_, w = random_forest_inputs(500 + M, kind, B, C, inner, T, depth, (M,), quantise=True)
    want = ho.forward(kind, x, thr, ord_, w)
    g = np.random.default_rng(7).standard_normal(want.shape).astype(np.float32)
    ref = ho.backward(kind, x, thr, ord_, w, g)
    sizes = ho.backward_magnitudes(kind, x, thr, ord_, w, g)
    # double precision on the same numbers: the oracle's sums in single precision are as good as the bar
    dx, dthr, dord, dw, dg = [a if a.dtype == torch.int64 else a.to(dtype) for a in dev(x, thr, ord_, w, g)]
    from hingetreefortorch_b200._ext import hingetree_cpp
    gx, gthr, _, gw = getattr(hingetree_cpp, kind + "_backward")(dx, True, dthr, True, dord, False, dw, True, dg)
    for got, r, s in zip((gx, gthr, gw), ref, sizes):
        assert grad_close(got, r, s)


@pytest.mark.parametrize("depth", [5, 8])
def test_terms_formed_in_the_reduction(depth):
    """One output per leaf, many samples: the expansion hands on the upstream gradient and the reduction forms the terms."""
    B, C, T = 65537 + 30, 20, 16
    x, thr, ord_, w = random_forest_inputs(400 + depth, "tree", B, C, (), T, depth, (), quantise=True)
    g = np.random.default_rng(6).standard_normal((B, T)).astype(np.float32)
    ref = ho.backward("tree", x, thr, ord_, w, g)
    sizes = ho.backward_magnitudes("tree", x, thr, ord_, w, g)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    f = _cabi.Forest("tree", dx, dw)
    assert f.saves_forward()
    for need in ((True, True, True), (True, True, False), (True, False, True)):
        f.forward(dx, dthr, dord, dw, save=True)
        for wanted, got, r, s in zip(need, f.backward(dx, dthr, dord, dw, dg, need=need, saved=True), ref, sizes):
            assert (got is None) if not wanted else grad_close(got, r, s)
